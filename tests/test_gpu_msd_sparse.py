"""MSD with origins further apart than the lags reach: the integer form stages the
frames that some lag reads and no others.  Tolerance as in the other MSD tests:
1e-12 relative against the oracle's running mean (lib/src/msd.cpp:70-118)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# N, frames, types, skip, lags, origins, first frame
CASES = [
    (70, 2000, 2, 50, 10, 39, 5),       # every origin in one tile
    (40, 3000, 1, 10, 9, 299, 0),       # the least gap
    (40, 3000, 3, 10, 10, 298, 1),      # none
    (13, 9200, 2, 30, 20, 305, 3),      # several tiles of origins
    (9, 9200, 2, 1500, 1400, 5, 100),   # long lags, few origins
    (5, 9000, 1, 2300, 2200, 3, 0),     # two origins a tile
    (33, 200, 4, 190, 3, 2, 0),
]


@pytest.mark.parametrize("cm", [False, True])
@pytest.mark.parametrize("case", CASES, ids=[str(i) for i in range(len(CASES))])
def test_sparse_origins(gpu_engine, oracle_mod, case, cm):
    N, T, nt, skip, lags, origins, primo = case
    rng = np.random.default_rng(3)
    pos = rng.uniform(-20, 20, (1, N, 3)) + np.cumsum(rng.normal(0, 0.1, (T, N, 3)), axis=0)
    tids = rng.permutation(np.arange(N) % nt).astype(np.int32)
    n = (origins - 1) * skip + 1
    assert lags <= n and lags + n + primo <= T
    box = np.zeros((T, 6))
    box[:, 3:6] = 50.0
    centres = oracle_mod.centres(pos, tids, nt)
    gpu_engine.set_frames(pos, box, tids, nt)
    gpu_engine.set_centres(centres)
    out = gpu_engine.msd(skip, lags, n, primo, cm, cm)
    ref = oracle_mod.msd(pos, tids, nt, skip, lags, n, primo, cm, cm, cm=centres)
    np.testing.assert_allclose(out, ref, rtol=1e-12, atol=0)
