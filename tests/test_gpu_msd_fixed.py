"""The integer form of the MSD where it can go wrong: more lags than threads,
tiles of origins, fewer atoms of a type than a group, types without atoms, lags
that do not fit (the FP64 form), coordinates far from zero and across it, and
displacements so small beside the coordinates that the FP64 form has to take
over.  Same tolerance as the FP64 form's test: 1e-12 relative against the
oracle's running mean (lib/src/msd.cpp:70-118), whose own error for these term
counts is below 1e-13."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def _walk(N, T, sigma, spread, offset=0.0, seed=1):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-spread, spread, size=(1, N, 3)) + offset
    return x + np.cumsum(rng.normal(0.0, sigma, size=(T, N, 3)), axis=0)


def _check(eng, oracle_mod, pos, tids, nt, skip, tmax, n, primo=0, cm=False):
    N = pos.shape[1]
    box = np.zeros((pos.shape[0], 6))
    box[:, 3:6] = 50.0
    centres = oracle_mod.centres(pos, tids, nt)
    eng.set_frames(pos, box, tids, nt)
    eng.set_centres(centres)
    out = eng.msd(skip, tmax, n, primo, cm, cm)
    ref = oracle_mod.msd(pos, tids, nt, skip, tmax, n, primo, cm, cm, cm=centres)
    present = np.bincount(tids, minlength=nt) > 0
    np.testing.assert_allclose(out[:, 0][:, present], ref[:, 0][:, present], rtol=RTOL, atol=0)
    if cm:
        np.testing.assert_allclose(out[:, 1][:, present], ref[:, 1][:, present], rtol=RTOL,
                                   atol=0)
    return out


# N, T, types, sigma, spread, offset, skip, tmax, n, primo
CASES = [
    (37, 1300, 2, 0.1, 20.0, 0.0, 7, 600, 600, 3),       # two passes over the lags
    (21, 6100, 3, 0.1, 20.0, 5.0, 1, 40, 6000, 0),       # tiles of origins
    (5, 4700, 1, 0.1, 20.0, 0.0, 2, 4500, 10, 0),        # lags that do not fit: FP64
    (200, 90, 40, 0.2, 10.0, 0.0, 3, 20, 60, 1),         # five atoms a type
    (17, 60, 17, 0.2, 10.0, -3.0, 1, 1, 50, 0),          # one atom a type, one lag
    (300, 80, 2, 1e-3, 10.0, 1e5, 2, 30, 40, 0),         # far from zero
    (300, 80, 2, 1e-6, 10.0, 0.0, 2, 30, 40, 0),         # tiny steps across zero: FP64
    (300, 80, 2, 1e3, 1e6, 0.0, 2, 30, 40, 0),           # long steps
]


@pytest.mark.parametrize("cm", [False, True])
@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_fixed_point_msd(gpu_engine, oracle_mod, case, cm):
    N, T, nt, sigma, spread, offset, skip, tmax, n, primo = case
    pos = _walk(N, T, sigma, spread, offset)
    tids = np.random.default_rng(2).permutation(np.arange(N) % nt).astype(np.int32)
    _check(gpu_engine, oracle_mod, pos, tids, nt, skip, tmax, n, primo, cm)


def test_atoms_at_rest_and_beside_large_coordinates(gpu_engine, oracle_mod):
    """Frozen atoms give exactly zero; atoms that move by 1e-4 near zero beside
    others at 1e5 keep the reference's precision (the FP64 form)."""
    pos = _walk(60, 50, 1e-4, 0.5)
    pos[:, :20] = pos[0, :20]
    pos[:, 20:40] += 1e5
    tids = (np.arange(60) // 20).astype(np.int32)
    out = _check(gpu_engine, oracle_mod, pos, tids, 3, 1, 20, 25)
    assert np.all(out[:, 0, 0] == 0.0)


def test_centres_that_are_not_finite_reach_the_result(gpu_engine, oracle_mod):
    pos = _walk(40, 30, 0.1, 5.0)
    tids = (np.arange(40) % 2).astype(np.int32)
    box = np.zeros((30, 6))
    box[:, 3:6] = 50.0
    centres = oracle_mod.centres(pos, tids, 2)
    centres[7, 1, 2] = np.nan
    gpu_engine.set_frames(pos, box, tids, 2)
    gpu_engine.set_centres(centres)
    out = gpu_engine.msd(1, 5, 10, 0, True, True)
    assert np.all(np.isfinite(out[:, :, 0])) and np.all(np.isnan(out[1:, :, 1]))
