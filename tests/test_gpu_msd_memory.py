"""The integer MSD's sums that do not fit the device (only their allocation fails,
ANALISI_GB300_FAIL_ALLOC=msd_sums): the FP64 form gives the results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_sums_where_the_integer_sums_do_not_fit(built_engine, monkeypatch):
    from analisi_gb300 import engine
    rng = np.random.default_rng(4)
    pos = rng.uniform(-20, 20, (1, 90, 3)) + np.cumsum(rng.normal(0, 0.1, (70, 90, 3)), axis=0)
    box = np.zeros((70, 6))
    box[:, 3:6] = 50.0
    with engine.Engine(0) as e:
        e.set_frames(pos, box, (np.arange(90) % 3).astype(np.int32), 3)
        monkeypatch.setenv("ANALISI_GB300_FAIL_ALLOC", "msd_sums")
        got = e.msd(2, 20, 50, 0).copy()
        assert e.stats()["rechecks"] == e.stats()["pairs"] == 20 * 25 * 90
        monkeypatch.delenv("ANALISI_GB300_FAIL_ALLOC")
        want = e.msd(2, 20, 50, 0)
        assert e.stats()["rechecks"] == 0
    # FP64 sums: 30 atoms and 25 origins, 50 units of 2^-53 at most (as derived where
    # the integer sums give way to them)
    np.testing.assert_allclose(got, want, rtol=50 * 2.0 ** -53, atol=0)
