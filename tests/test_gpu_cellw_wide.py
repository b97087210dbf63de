"""Histograms that leave the warp-streamed cell-list kernel one CTA per SM: the
CTA of 32 warps (and, past its room, the CTA of 16), every kind of rmin, counts
per partition, orthorhombic and triclinic.  Counts equal the oracle's."""
import numpy as np
import pytest

from analisi_gb300 import engine, workloads

pytestmark = pytest.mark.gpu

# types, bins, rmin, triclinic, partitions
CASES = [
    (5, 500, 0.0, False, 1),    # 60 KB of cells: one CTA of 32 warps
    (5, 500, 0.8, True, 1),
    (5, 500, -0.6, False, 1),
    (3, 301, 0.0, False, 5),    # five partitions of 14 KB in one histogram
    (6, 600, 0.0, False, 1),    # 101 KB: one CTA of 16 warps
    (6, 870, 0.0, False, 1),    # 146 KB: the last of them
    (6, 960, 0.0, False, 1),    # 161 KB: no room for 16 warps, the all-pairs kernel
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(str(x) for x in c))
def test_large_histograms(gpu_engine, oracle_mod, case):
    nt, nbin, rmin, tric, nparts = case
    N, L, rmax = 2600, 30.0, 5.0
    counts = [N // nt] * nt
    counts[0] += N - sum(counts)
    w = workloads.small_case(nt + nbin, N, 7, L, 0.2, counts, tric=tric, wrap_into_cell=tric)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"], triclinic=tric)
    args = (rmin, rmax, nbin, 2, 2, 1, 5, 1)
    got = gpu_engine.run(*args, nparts=nparts)
    assert gpu_engine.stats()["kernel_used"] == (1 if nbin == 960 else 5)
    want = oracle_mod.gofrt_counts(w["positions"], w["boxes"], w["type_ids"], nt, rmin, rmax, nbin,
                                   2, nparts, 2, 1, 5, 1, tric=tric, per_thread=nparts > 1)
    np.testing.assert_array_equal(got, want)


def test_forced_kernel_keeps_its_limit(gpu_engine):
    """kernel="cellw" refuses a histogram it refused before AUTO took it."""
    w = workloads.small_case(3, 2600, 3, 30.0, 0.2, [434, 434, 433, 433, 433, 433])
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"])
    with pytest.raises(engine.GofrError):
        gpu_engine.run(0.0, 5.0, 600, 1, 1, 1, 2, 0, kernel="cellw")


@pytest.mark.parametrize("N,L,kernel,rmin,rmax", [
    (129, 10.0, "f32", 4.0, 4.004), (250, 10.0, "f32", 4.0, 4.004), (129, 10.0, "f32", -1e-4, 1e-4),
    (250, 10.0, "f32", -1e-4, 1e-4), (2600, 30.0, "cellw", 4.0, 4.004)])
def test_bins_finer_than_the_margin(gpu_engine, oracle_mod, N, L, kernel, rmin, rmax):
    """Bins so fine that every pair is recomputed: the lanes without an atom of
    the last chunk are not, the pairs clamped to the row's ends are."""
    w = workloads.small_case(N, N, 5, L, 0.2, [N - N // 3, N // 3])
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"])
    got = gpu_engine.run(rmin, rmax, 500, 2, 1, 1, 4, 0, kernel=kernel)
    want = oracle_mod.gofrt_counts(w["positions"], w["boxes"], w["type_ids"], 2, rmin, rmax, 500,
                                   2, 1, 1, 1, 4, 0)
    np.testing.assert_array_equal(got, want)
    assert want.sum() > 0 or rmin < 0
