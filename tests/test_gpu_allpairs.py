"""The kernels that bin a pair where they find it, at the sizes where their
units can go wrong: atom counts around the groups of 32 and 64 first atoms and
the chunks of 128 second atoms, jobs of few (lag, origin) pairs (units split
over the second atoms), many types in a group, reference partitions shorter
than a group, several windows in one launch, rmin zero, positive and negative,
minimum images that are not certain, and batches that mix them.  Counts equal
the oracle's."""
import numpy as np
import pytest

from analisi_gb300 import engine, workloads

pytestmark = pytest.mark.gpu


def _case(N, L, ntypes, tric=False, seed=None, T=9):
    counts = [N // ntypes] * ntypes
    counts[0] += N - sum(counts)
    return workloads.small_case(seed or N, N, T, L, 0.2, counts, tric=tric, wrap_into_cell=tric)


def _ref(oracle_mod, w, p, threads=1, per_thread=False):
    return oracle_mod.gofrt_counts(w["positions"], w["boxes"], w["type_ids"], w["ntypes"], p["rmin"],
                                   p["rmax"], p["nbin"], p["tmax"], threads, p["skip"], p["every"],
                                   p["ntimesteps"], p["primo"], tric=w["triclinic"],
                                   per_thread=per_thread)


def _p(rmin, rmax, nbin=37, tmax=3, skip=2, every=1, ntimesteps=5, primo=1):
    return dict(rmin=rmin, rmax=rmax, nbin=nbin, tmax=tmax, skip=skip, every=every,
                ntimesteps=ntimesteps, primo=primo)


# N, L, types, triclinic, rmin, rmax (the last two rows: images near L/2 within rmax)
CASES = [
    (31, 9.0, 1, False, 0.0, 4.0), (64, 9.0, 3, False, 0.4, 4.0), (65, 9.0, 2, True, 0.0, 3.9),
    (127, 10.0, 5, False, -0.7, 4.0), (128, 10.0, 2, False, 0.0, 4.9), (129, 10.0, 40, True, 0.3, 4.0),
    (2305, 24.0, 3, False, 0.0, 11.5), (200, 9.0, 2, False, 0.0, 5.5), (150, 9.0, 3, True, -0.4, 5.0),
]


@pytest.mark.parametrize("case", CASES, ids=[f"n{c[0]}" for c in CASES])
def test_group_and_chunk_edges(gpu_engine, oracle_mod, case):
    N, L, nt, tric, rmin, rmax = case
    w = _case(N, L, nt, tric)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"], triclinic=tric)
    for p in (_p(rmin, rmax), _p(rmin, rmax, tmax=1, skip=5)):
        args = [p[k] for k in ("rmin", "rmax", "nbin", "tmax", "skip", "every", "ntimesteps",
                               "primo")]
        got = gpu_engine.run(*args, kernel="f32")
        np.testing.assert_array_equal(got, _ref(oracle_mod, w, p))
        parts = 1 + N // 25 if N < 1000 else 7
        got = gpu_engine.run(*args, kernel="f32", nparts=parts)
        np.testing.assert_array_equal(got, _ref(oracle_mod, w, p, parts, True))
    p = _p(rmin, rmax, tmax=2, ntimesteps=3)
    got = gpu_engine.run_windows(rmin, rmax, p["nbin"], 2, 2, 1, 3, [4, 0, 2], kernel="f32",
                                 nparts=3)
    for k, first in enumerate([4, 0, 2]):
        np.testing.assert_array_equal(got[k], _ref(oracle_mod, w, dict(p, primo=first), 3, True))


@pytest.mark.parametrize("rmin", [0.0, 0.6, -0.9])
def test_cell_lists_with_every_kind_of_rmin(gpu_engine, oracle_mod, rmin):
    w = _case(2300, 27.0, 3)
    p = _p(rmin, 5.0)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"])
    got = gpu_engine.run(p["rmin"], p["rmax"], p["nbin"], p["tmax"], p["skip"], p["every"],
                         p["ntimesteps"], p["primo"], kernel="cellw")
    assert gpu_engine.stats()["kernel_used"] == 5
    np.testing.assert_array_equal(got, _ref(oracle_mod, w, p))


@pytest.mark.parametrize("rmin", [0.0, -0.5])
def test_batch_of_every_kind(gpu_engine, oracle_mod, rmin):
    """Members with and without certain images, of several bin maps and lag counts
    (rmin = 0 alone takes the kernel without the general bin map)."""
    members = [(_case(40, 6.0, 2), _p(0.0, 4.5, nbin=11)), (_case(700, 19.0, 4), _p(rmin, 7.0)),
               (_case(333, 14.0, 1), _p(0.0, 6.0, nbin=90, tmax=4, skip=1)),
               (_case(3000, 31.0, 2), _p(0.0, 4.5))]
    gpu_engine.batch_set([dict(positions=w["positions"], boxes=w["boxes"], type_ids=w["type_ids"],
                               ntypes=w["ntypes"],
                               params=engine.make_params(*[p[k] for k in (
                                   "rmin", "rmax", "nbin", "tmax", "skip", "every", "ntimesteps",
                                   "primo")])) for w, p in members])
    for use_graph in (True, False):
        for got, (w, p) in zip(gpu_engine.batch_run(use_graph=use_graph), members):
            np.testing.assert_array_equal(got, _ref(oracle_mod, w, p))


# N, L, types, triclinic, rmax, bins, partitions, kernel (40: more partitions than
# one histogram holds, in a box where the all-pairs kernel is the cheaper one
# then, and in one where it is not; 700: more partitions than atoms of a warp block)
@pytest.mark.parametrize("case", [(2300, 27.0, 3, False, 5.0, 37, 4, 5),
                                  (2301, 27.0, 3, False, 5.0, 400, 40, 1),
                                  (6001, 45.0, 3, False, 5.0, 400, 40, 5),
                                  (2099, 26.0, 1, False, 4.0, 20, 700, 5),
                                  (4100, 33.0, 2, True, 6.0, 50, 3, 5)],
                         ids=["4", "40-allpairs", "40", "700", "tric"])
def test_cell_lists_per_partition(gpu_engine, oracle_mod, case):
    N, L, nt, tric, rmax, nbin, parts, kernel = case
    w = _case(N, L, nt, tric)
    p = _p(0.0, rmax, nbin=nbin)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], w["ntypes"], triclinic=tric)
    args = [p[k] for k in ("rmin", "rmax", "nbin", "tmax", "skip", "every", "ntimesteps", "primo")]
    got = gpu_engine.run(*args, nparts=parts)
    assert gpu_engine.stats()["kernel_used"] == kernel
    np.testing.assert_array_equal(got, _ref(oracle_mod, w, p, parts, True))
    got = gpu_engine.run_windows(p["rmin"], rmax, nbin, 2, 2, 1, 3, [3, 0], nparts=parts)
    for k, first in enumerate([3, 0]):
        np.testing.assert_array_equal(
            got[k], _ref(oracle_mod, w, dict(p, tmax=2, ntimesteps=3, primo=first), parts, True))
    # a forced cell-list kernel still refuses partitions
    with pytest.raises(engine.GofrError):
        gpu_engine.run(*args, kernel="cellw", nparts=parts)


def test_tuned_windows_sample_the_first_window(gpu_engine, oracle_mod):
    """The tuner of a run over windows samples the first window: the parameters'
    own first frame, here past the end, is not one of them."""
    import ctypes
    w = workloads.small_case(83, 6000, 6, 42.0, 0.1, [4000, 2000], rmin=0.0, rmax=4.0, nbin=37,
                             tmax=2, skip=1, every=1, ntimesteps=3, primo=0)
    gpu_engine.set_frames(w["positions"], w["boxes"], w["type_ids"], 2)
    p = engine.make_params(0.0, 4.0, 37, 2, 1, 1, 3, 1 << 40, "tuned")
    primos = np.array([2, 0], dtype=np.uint64)
    out = np.zeros(2 * 2 * 6 * 37, dtype=np.uint64)
    as_u64 = ctypes.POINTER(ctypes.c_ulonglong)
    gpu_engine._check(gpu_engine.L.gofr_run_windows(
        gpu_engine._ctx, ctypes.byref(p), 2, primos.ctypes.data_as(as_u64),
        out.ctypes.data_as(as_u64)))
    # an eightieth of the pairs is near: all pairs would be an order slower
    assert gpu_engine.stats()["kernel_used"] in (3, 5)
    for k, primo in enumerate((2, 0)):
        want = oracle_mod.gofrt_counts(w["positions"], w["boxes"], w["type_ids"], 2, 0.0, 4.0, 37,
                                       2, 8, 1, 1, 3, primo)
        np.testing.assert_array_equal(out.reshape(2, *want.shape)[k], want)
