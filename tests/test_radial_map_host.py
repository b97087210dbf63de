"""The bin map of the kernels that bin a pair where they find it, checked on
the CPU: pairs placed within a few margins of bin edges are put through the
kernel's FP32 operations in numpy (the warp-streamed kernel's: coordinates
reduced into the cell, the neighbour moved by the FP32 image vector; the
all-pairs kernel's: both atoms moved into the box, |d| or L - |d|; triclinic, the
FP32 minimum image), with the hardware rsqrt at both ends of
its stated error and at its centre.  Every pair the map calls certain must be
in the reference's bin (lib/src/gofrt.cpp:104,114-118 on its FP64 minimum
image), and every pair the reference counts must come out inside the map's
window; boxes shifted, triclinic and far unwrapped, rmin zero, positive and
negative, wide and very narrow bins."""
import math

import numpy as np
import pytest

from analisi_gb300 import engine

from test_cell_bound_host import fma32, reduce_into_cell, ref_d2, ref_image

MAGIC = np.float32(12582912.0)
f32 = np.float32

# L3, tilt {xy, xz, yz}, lo, lattice vectors out, (rmin, rmax, nbin), kernel
CASES = [
    ((54.72, 54.72, 54.72), (0, 0, 0), (0.0, 0.0, 0.0), 0, (0.0, 12.0, 400), "cellw"),
    ((54.72, 54.72, 54.72), (0, 0, 0), (0.0, 0.0, 0.0), 0, (0.0, 12.0, 400), "f32"),
    ((109.4, 109.4, 109.4), (0, 0, 0), (0.0, 0.0, 0.0), 0, (0.0, 10.0, 250), "cellw"),
    ((70.0, 70.0, 70.0), (21.0, 14.0, 7.0), (0.0, 0.0, 0.0), 0, (0.0, 15.0, 500), "cellw"),
    ((70.0, 70.0, 70.0), (21.0, 14.0, 7.0), (0.0, 0.0, 0.0), 0, (0.0, 15.0, 500), "f32"),
    ((26.0, 31.0, 35.0), (-8.0, 11.0, -13.0), (-3.0, 2.5, 7.0), 3, (0.7, 6.0, 53), "cellw"),
    ((27.0, 25.0, 29.0), (0, 0, 0), (4.0, -6.0, 1.5), 40, (0.3, 5.5, 97), "cellw"),
    ((22.0, 22.0, 22.0), (0, 0, 0), (-3.0, 0.0, 9.0), 1, (0.7, 3.5, 200), "f32"),
    ((28.0, 28.0, 28.0), (0, 0, 0), (0.0, 0.0, 0.0), 0, (0.0, 13.5, 300), "f32"),
    ((28.0, 28.0, 28.0), (0, 0, 0), (0.0, 0.0, 0.0), 2, (-1.0, 5.0, 37), "f32"),
    ((28.0, 28.0, 28.0), (0, 0, 0), (0.0, 0.0, 0.0), 0, (0.0, 5.0, 2000), "cellw"),
]


def allpairs_d(xi, xj, lo3, hi3, L, tilt, tric):
    shift = 0.5 * lo3 + 0.5 * hi3
    L32, inv = L.astype(f32), (1.0 / L).astype(f32)
    t32 = np.array(tilt, dtype=f32)
    one = np.ones(len(xi), dtype=f32)

    def wrap(v, ax):
        return (fma32(v, inv[ax] * one, MAGIC * one) - MAGIC).astype(f32)

    ai, aj = (xi - shift).astype(f32), (xj - shift).astype(f32)
    if not tric:  # both atoms into the box, then |d| or L - |d|
        d = np.empty_like(ai)
        for ax in range(3):
            wi = fma32(wrap(ai[:, ax], ax), -L32[ax] * one, ai[:, ax])
            wj = fma32(wrap(aj[:, ax], ax), -L32[ax] * one, aj[:, ax])
            a = np.abs((wi - wj).astype(f32))
            d[:, ax] = np.minimum(a, (L32[ax] - a).astype(f32))
        return d
    d = (ai - aj).astype(f32)
    k = wrap(d[:, 2], 2)
    d[:, 2] = fma32(k, -L32[2] * one, d[:, 2])
    d[:, 1] = fma32(k, -t32[2] * one, d[:, 1])
    d[:, 0] = fma32(k, -t32[1] * one, d[:, 0])
    k = wrap(d[:, 1], 1)
    d[:, 1] = fma32(k, -L32[1] * one, d[:, 1])
    d[:, 0] = fma32(k, -t32[0] * one, d[:, 0])
    k = wrap(d[:, 0], 0)
    d[:, 0] = fma32(k, -L32[0] * one, d[:, 0])
    return d


def cellw_d(xi, xj, d_ref, tab, lo, L, tilt):
    wi, wj = reduce_into_cell(xi, lo, L, tilt), reduce_into_cell(xj, lo, L, tilt)
    c = lo + L / 2
    D = (wi - wj) - d_ref
    sz = np.rint(D[:, 2] / L[2])
    sy = np.rint((D[:, 1] - sz * tilt[2]) / L[1])
    sx = np.rint((D[:, 0] - sz * tilt[1] - sy * tilt[0]) / L[0])
    sh = tab["shift"][((sx + 2) + 5 * (sy + 2) + 25 * (sz + 1)).astype(int)]
    b = ((wj - c).astype(f32) + sh).astype(f32)
    return ((wi - c).astype(f32) - b).astype(f32)


@pytest.mark.parametrize("case", CASES, ids=[f"{i}-{c[5]}" for i, c in enumerate(CASES)])
def test_certain_pairs_are_in_the_reference_bin(built_engine, case):
    L3, tilt, lo, out, (rmin, rmax, nbin), kernel = case
    tric = any(t != 0 for t in tilt)
    L, lo = np.array(L3), np.array(lo)
    H = np.array([[L[0], 0, 0], [tilt[0], L[1], 0], [tilt[1], tilt[2], L[2]]], dtype=float)
    rng = np.random.default_rng(5)
    n = 100000
    dr = (rmax - rmin) / nbin
    xi = rng.random((n, 3)) @ H + lo + rng.integers(-out, out + 1, (n, 3)) @ H
    v = rng.normal(size=(n, 3))
    # half of the pairs near a bin edge (rmin, rmax and -rmin among them), half anywhere
    r = rmin + dr * rng.integers(0, nbin + 1, n) + rng.normal(size=n) * 6e-5
    r[: n // 2] = rmax * 1.01 * rng.random(n // 2) ** (1 / 3)
    r[-500:] = abs(rmin) + rng.normal(size=500) * 6e-5
    r[-1000:-500] = rmax + rng.normal(size=500) * 6e-5
    v *= (np.abs(r) / np.linalg.norm(v, axis=1))[:, None]
    xj = xi - v + rng.integers(-out - 1, out + 2, (n, 3)) @ H
    d_ref = ref_image(xi - xj, L, tilt)
    s_ref = ref_d2(d_ref)
    keep = np.sqrt(s_ref) < rmax * 1.02
    xi, xj, d_ref, s_ref = xi[keep], xj[keep], d_ref[keep], s_ref[keep]
    allx = np.concatenate([xi, xj])
    internal = list(lo) + list(L / 2) + (list(tilt) if tric else [])
    args = (internal, tric, allx.min(0), allx.max(0))
    natoms = 20000
    p = engine.make_params(rmin, rmax, nbin, 2, 1, 1, 4, 0, kernel=kernel)
    m = engine.radial_query(*args, natoms, 2, p)
    plan = engine.plan_query(*args, natoms, 2, p)
    # the reference's bin (-1: not counted)
    q = ((np.sqrt(s_ref) - rmin) / dr).astype(f32)
    fl = np.floor(q)
    ok = (s_ref <= rmax * rmax) & (s_ref >= rmin * rmin) & (fl >= 0) & (fl < nbin)
    want = np.where(ok, fl, -1).astype(int)
    if kernel == "cellw":
        tab = engine.cellw_tables(*args, rmax, list(plan["cells"]))
        d = cellw_d(xi, xj, d_ref, tab, lo, L, tilt)
    else:
        d = allpairs_d(xi, xj, allx.min(0), allx.max(0), L, tilt, tric)
    one = np.ones(len(d), dtype=f32)
    d2 = fma32(d[:, 2], d[:, 2], fma32(d[:, 1], d[:, 1], fma32(d[:, 0], d[:, 0], f32(1e-30) * one)))
    for s in (-1.0, 0.0, 1.0):
        rs = (1.0 / np.sqrt(d2.astype(np.float64)) * (1.0 + s * 2.0 ** -22.9)).astype(f32)
        qq = fma32((d2 * m["inv_dr"]).astype(f32), rs, m["q_off"] * one)
        t = (qq + MAGIC).astype(f32)
        bin_ = (t.astype(np.float64) - float(MAGIC)).astype(int)
        certain = np.abs((qq - (t - MAGIC).astype(f32)).astype(f32)) <= m["lim"]
        if rmin < 0:
            certain &= (t >= m["t_ok"]) | (t < m["t_lo"])
        got = np.where((bin_ >= 0) & (bin_ < nbin) & (t >= m["t_lo"]), bin_, -1)
        np.testing.assert_array_equal(got[certain], want[certain])
        # nothing the reference counts leaves the window
        assert np.all((t[want >= 0] >= m["t_lo"]) & (t[want >= 0] <= m["t_hi"]))
        # most pairs are certain (bins far wider than the margin), and the margin
        # is not many times what these pairs needed
        anywhere = np.zeros(len(r), dtype=bool)
        anywhere[: n // 2] = True
        if nbin < 1000:
            assert certain[anywhere[keep]].mean() > 0.98
    assert 0.0 < m["lim"] < 0.5 and m["lim_self"] < 0.5
