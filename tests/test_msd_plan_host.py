"""How the integer MSD lays a job out (host planner): whatever the origins' spacing,
its threads have work and its tiles hold only frames that some lag reads."""
import pytest

from analisi_gb300 import engine

THREADS, ENTRIES = 512, 4480


@pytest.mark.parametrize("skip", [1, 2, 9, 10, 11, 60, 500, 100000])
@pytest.mark.parametrize("lags", [1, 3, 10, 50, 100, 600, 2000])
@pytest.mark.parametrize("origins", [1, 2, 7, 40, 200, 3000])
@pytest.mark.parametrize("natoms", [1, 50, 3000, 200000])
def test_threads_and_frames(built_engine, natoms, lags, origins, skip):
    p = engine.msd_plan_query(natoms, lags, origins, skip)
    if 8 * skip > 5 * lags and lags >= 32 and origins * lags >= 4 * 152:
        assert p is None  # FP64 sums
        return
    tile = p["origins"]
    apart = skip >= lags or origins == 1  # no frame is in the lags of two origins
    assert 1 <= tile <= origins and p["tiles"] == -(-origins // tile)
    assert p["frames"] == (tile - 1) * skip + lags
    assert tile == 1 if apart else p["frames"] <= tile * lags
    assert p["frames"] * p["atoms"] <= ENTRIES and 3 * p["atoms"] <= THREADS
    assert p["lags"] == min(lags, THREADS)
    # a thread per (lag, phase of the tile's origins, or of its atoms); nearly all of
    # them where there are as many
    phases = p["atoms"] if apart else tile
    assert p["phases"] == min(THREADS // p["lags"], phases)
    assert apart or p["phases"] * p["lags"] > THREADS // 2 or tile == origins
