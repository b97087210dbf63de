"""The all-pairs kernel where few pairs are within rmax: 64 pairs of a first atom
without such a pair are passed over.  Counts against the oracle just below and
just above the shares from which every pair is binned, with empty and crowded
groups, every kind of bin map (rmin zero, positive, negative), triclinic boxes and
boxes that change from frame to frame."""
import numpy as np
import pytest

from analisi_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("natoms", [127, 300, 1000])
@pytest.mark.parametrize("share", [1e-5, 0.0099, 0.0101, 0.0139, 0.0141])
@pytest.mark.parametrize("rmin", [0.0, 0.4, -0.5])
@pytest.mark.parametrize("tric", [False, True])
@pytest.mark.parametrize("heaps", [False, True])
def test_counts_equal_the_oracle(gpu_engine, oracle_mod, natoms, share, rmin, tric, heaps):
    L = 30.0
    rmax = L * (share * 3.0 / (4.0 * np.pi)) ** (1.0 / 3.0)
    if rmin > 0.0:
        rmin *= rmax
    nbin = 20
    w = workloads.small_case(7, natoms, 6, L, 0.1, [natoms // 2, natoms - natoms // 2], rmin=rmin,
                             rmax=rmax, nbin=nbin, tmax=3, skip=1, every=1, ntimesteps=3, primo=0)
    pos = w["positions"].copy()
    if heaps:  # the first and last atoms in heaps of the size of rmax
        pos[:, :20] = pos[:, :1] + 0.5 * rmax * np.random.default_rng(1).normal(size=(6, 20, 3))
        pos[:, -9:] = pos[:, -1:]
    box = np.zeros((6, 9 if tric else 6))
    box[:, 3:6] = (L / 2) * (1.0 + 1e-3 * np.arange(6))[:, None]
    if tric:
        box[:, 6:] = [0.2 * L, 0.1 * L, 0.1 * L]
    args = (rmin, rmax, nbin, 3, 1, 1, 3, 0)
    gpu_engine.set_frames(pos, box, w["type_ids"], 2)
    got = gpu_engine.run(*args, kernel="auto")
    assert gpu_engine.stats()["kernel_used"] == 1
    ref = oracle_mod.gofrt_counts(pos, box, w["type_ids"], 2, rmin, rmax, nbin, 3, 8, 1, 1, 3, 0)
    np.testing.assert_array_equal(got, ref)
