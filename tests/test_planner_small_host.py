"""Where AUTO begins to take cell lists for small trajectories (host planner):
from 2048 atoms for any job, from 1024 for jobs of 2^28 ordered pairs."""
import pytest

from analisi_gb300 import engine

F32, CELLW = 1, 5


# atoms, lags, origins, kernel: 256 (lag, origin) frames of 1024 atoms are 2^28 pairs
@pytest.mark.parametrize("natoms,lags,origins,kernel", [
    (2048, 2, 2, CELLW), (2047, 2, 2, F32), (2047, 8, 9, CELLW),
    (1024, 16, 16, CELLW), (1024, 15, 17, F32), (1023, 60, 40, F32)])
@pytest.mark.parametrize("tric", [False, True])
@pytest.mark.parametrize("every", [1, 3])
def test_small_trajectories(built_engine, natoms, lags, origins, kernel, tric, every):
    L = 32.0
    box = [0.0] * 3 + [L / 2] * 3 + ([0.2 * L, 0.1 * L, 0.1 * L] if tric else [])
    p = engine.make_params(0.0, 4.0, 100, lags * every, 3, every, 3 * origins * every, 0)
    p.skip = 3 * every
    got = engine.plan_query(box, tric, [0.0] * 3, [L] * 3, natoms, 2, p)
    assert got["kernel"] == kernel
