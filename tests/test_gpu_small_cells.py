"""Cell lists for trajectories of 1024 to 2047 atoms, as AUTO takes them for jobs
large enough: counts equal the oracle's, single runs, partitions and windows."""
import numpy as np
import pytest

from analisi_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L,tric,parts", [(1024, 26.0, False, 1), (1025, 30.0, True, 1),
                                            (1501, 28.0, False, 3), (2047, 33.0, True, 1)])
def test_small_boxes(gpu_engine, oracle_mod, N, L, tric, parts):
    w = workloads.small_case(N, N, 35, L, 0.2, [N - 300, 200, 100], tric=tric, wrap_into_cell=tric)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], 3, triclinic=tric)
    tmax, n, primo = 16, 17, 1
    args = (0.0, 4.5, 90, tmax, 1, 1, n)
    got = gpu_engine.run(*args, primo, nparts=parts)
    assert gpu_engine.stats()["kernel_used"] == 5

    def want(first):
        return oracle_mod.gofrt_counts(w["positions"], w["boxes"], w["type_ids"], 3, 0.0, 4.5, 90,
                                       tmax, parts if parts > 1 else 8, 1, 1, n, first, tric=tric,
                                       per_thread=parts > 1)
    np.testing.assert_array_equal(got, want(primo))
    got = gpu_engine.run_windows(*args, [2, 0], nparts=parts)
    np.testing.assert_array_equal(got[1], want(0))
