"""Accuracy of the MSD against exact rational arithmetic where a fixed unit could
cost bits: atoms near zero beside large coordinates, windows within much longer
or jumping trajectories, types held still.

Tolerance, relative: what FP64 sums may be off by (a displacement rounded and
squared 2, the block's sum 13, three FMAs per 256 atoms, an addition per origin
and a division, in units of 2^-53) plus the bound up to which the integer sums
are kept (32 of these units) and their two roundings."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(pos, atoms, skip, leff, n, primo, centre=None):
    """Mean over origins and atoms of the squared displacement, per lag."""
    x = [[[Fraction(float(v)) for v in row] for row in frame] for frame in pos[:, atoms]]
    if centre is not None:
        x = [[[v - Fraction(float(c)) for v, c in zip(row, cm)] for row in frame]
             for frame, cm in zip(x, centre)]
    out = []
    for lag in range(leff):
        s = Fraction(0)
        for o in range(primo, primo + n, skip):
            for a, b in zip(x[o], x[o + lag]):
                s += sum((p - q) ** 2 for p, q in zip(a, b))
        out.append(s / (len(atoms) * len(range(primo, primo + n, skip))))
    return out


def _check(eng, pos, tids, nt, skip, leff, n, primo=0, cm=False):
    box = np.zeros((pos.shape[0], 6))
    box[:, 3:6] = 100.0
    eng.set_frames(pos, box, tids.astype(np.int32), nt)
    centres = None
    if cm:
        centres = np.stack([pos[:, tids == k].mean(axis=1) for k in range(nt)], axis=1)
        eng.set_centres(centres)
    got = eng.msd(skip, leff, n, primo, False, cm)[:, 0]
    for k in range(nt):
        atoms = np.flatnonzero(tids == k)
        origins = len(range(0, n, skip))
        tol = (16 + origins + 3 * -(-len(atoms) // 256) + 32 + 2) * 2.0 ** -53
        want = _exact(pos, atoms, skip, leff, n, primo, centres[:, k] if cm else None)
        for lag in range(leff):
            assert abs(Fraction(float(got[lag, k])) - want[lag]) <= Fraction(tol) * want[lag]


def _walk(rng, T, N, sigma):
    return np.cumsum(rng.normal(0.0, sigma, (T, N, 3)), axis=0)


@pytest.mark.parametrize("cm", [False, True])
@pytest.mark.parametrize("seed", range(6))
def test_tracers_near_the_origin_beside_a_large_box(gpu_engine, seed, cm):
    rng = np.random.default_rng(seed)
    pos = _walk(rng, 50, 40, 0.009) + rng.uniform(-64.0, 64.0, (1, 40, 3))
    few = 2 if cm else 1
    pos[:, :few] = _walk(rng, 50, few, 0.009) + rng.uniform(-0.2, 0.2, (1, few, 3))
    _check(gpu_engine, pos, (np.arange(40) >= few).astype(int), 2, 1, 6, 40, cm=cm)


@pytest.mark.parametrize("seed", range(3))
@pytest.mark.parametrize("skip,leff,n,primo,jump", [
    (12, 6, 240, 3, 100.0),    # origins apart, jumps between them
    (7, 6, 140, 0, 0.3),       # every frame in one extent
    (2, 5, 20, 30, 1.0e4),     # a window of a longer trajectory that jumps later
    (5, 5, 5, 0, 1.0),         # one origin
])
def test_windows_of_longer_trajectories(gpu_engine, seed, skip, leff, n, primo, jump):
    rng = np.random.default_rng(seed)
    pos = _walk(rng, 260, 9, 0.003) + rng.uniform(-1.0, 1.0, (1, 9, 3))
    late = np.arange(260) >= 80 if jump > 1e3 else (np.arange(260) - primo) % 12 >= 8
    pos[late, ::2] += jump
    _check(gpu_engine, pos, np.arange(9) % 3, 3, skip, leff, n, primo)


@pytest.mark.parametrize("scale", [1e-60, 1e-12, 1.0, 1e25, 1e120])
def test_held_still_and_other_scales(gpu_engine, scale):
    """A type at rest, one that oscillates by the last bit near zero, one that
    moves; coordinates beyond the range of the FP32 frames."""
    rng = np.random.default_rng(5)
    pos = _walk(rng, 30, 12, 0.05) + rng.uniform(-3.0, 3.0, (1, 12, 3))
    pos[:, :4] = pos[0, :4]
    pos[:, 4:8] = pos[0, 4:8] * 2.0 ** -40
    pos[::2, 4:8] = np.nextafter(pos[::2, 4:8], 1.0)
    _check(gpu_engine, pos * scale, np.arange(12) // 4, 3, 2, 7, 20)


def test_fp64_sums_only_where_lost_bits_could_show(gpu_engine):
    """A type that oscillates by the last bit near zero is summed in FP64; the others,
    one of which is at rest and one moves by 0.003 a step in a box of 200, are not
    (the displacements summed in FP64 are in the statistics)."""
    rng = np.random.default_rng(7)
    pos = _walk(rng, 30, 40, 0.003) + rng.uniform(-100.0, 100.0, (1, 40, 3))
    pos[:, :10] = pos[0, :10]
    _check(gpu_engine, pos, np.arange(40) // 10, 4, 2, 7, 20)
    assert gpu_engine.stats()["rechecks"] == 0
    pos[:, 10:20] = pos[0, 10:20] * 2.0 ** -40
    pos[::2, 10:20] = np.nextafter(pos[::2, 10:20], 1.0)
    _check(gpu_engine, pos, np.arange(40) // 10, 4, 2, 7, 20)
    assert gpu_engine.stats()["rechecks"] == 10 * 10 * 6  # its atoms, origins, lags 1 to 6
