"""The trimmed rows of the warp-streamed cell-list kernel, on the CPU.

A row of a warp block's neighbourhood keeps only the cells within reach at the
row's distance in y and z (gofr_cellw_row: the host and the kernel call the
same function).  Every warp block of a grid is walked as the kernel walks it
and the pairs reached are compared with a brute-force evaluation of the
reference's minimum image (lib/include/basetrajectory.h:224-268): each pair
within rmax exactly once.  Atoms on cell faces and box faces, cells finer in x,
tilts of both signs, shifted boxes, blocks of several cells."""
import functools
import math

import numpy as np
import pytest

from analisi_gb300 import engine
from test_cellw_geometry import BOXES, lattice_case, reduce_into_cell, ref_image


@pytest.mark.parametrize("faces", [False, True], ids=["random", "faces"])
@pytest.mark.parametrize("m,fx,wblk", [(1, 1, (1, 1, 1)), (1, 8, (1, 1, 1)), (2, 4, (1, 1, 1)),
                                       (2, 2, (2, 1, 2)), (3, 2, (2, 2, 1))])
@pytest.mark.parametrize("box", BOXES, ids=[str(i) for i in range(len(BOXES))])
def test_trimmed_rows_reach_every_pair_once(built_engine, box, m, fx, wblk, faces):
    L3, tilt, lo, unwrap, rmax = box
    tric = any(t != 0.0 for t in tilt)
    ibox = [*lo, *(v / 2 for v in L3)] + (list(tilt) if tric else [])
    coarse = [math.floor(L3[k] * m / (rmax * (1 + 1e-6))) for k in range(3)]
    assert all(n >= 2 * m + 1 for n in coarse)
    nc = [coarse[0] * fx, coarse[1], coarse[2]]
    w = [wblk[0] * fx, wblk[1], wblk[2]]
    N = 500
    pos = lattice_case(31 + m, N, L3, tilt, lo, unwrap)
    if faces:  # half the atoms on faces of the fine grid (and of the box)
        f = np.floor((pos[:N // 2] - lo) / L3 * nc) / nc
        pos[:N // 2] = f * L3 + np.array(lo)
        # and pairs that lie rmax apart along x, a hair inside
        pos[N // 2:N // 2 + 50] = pos[:50] + [rmax * (1 - 1e-12), 0.0, 0.0]
    mn, mx = pos.min(0), pos.max(0)
    tab = engine.cellw_tables(ibox, tric, mn, mx, rmax, nc)
    assert tab is not None
    H = np.array([[L3[0], 0, 0], [tilt[0], L3[1], 0], [tilt[1], tilt[2], L3[2]]])
    wr = reduce_into_cell(pos, np.array(lo), np.array(L3), tilt, tric)
    cell = np.clip(np.floor((wr - lo) / L3 * nc).astype(int), 0, np.array(nc) - 1)
    cid = (cell[:, 2] * nc[1] + cell[:, 1]) * nc[0] + cell[:, 0]
    order = np.argsort(cid, kind="stable")
    start = np.searchsorted(cid[order], np.arange(nc[0] * nc[1] * nc[2] + 1))

    @functools.lru_cache(None)
    def row_range(cn, row):
        return engine.cellw_row(ibox, tric, mn, mx, rmax, nc, cn, row)

    got = np.zeros((N, N), dtype=int)
    kept = whole = 0
    nz_lo, nz_hi = tab["nz"]
    for z0 in range(0, nc[2], w[2]):
        for y0 in range(0, nc[1], w[1]):
            for x0 in range(0, nc[0], w[0]):
                c0 = (x0, y0, z0)
                cn = tuple(min(w[k], nc[k] - c0[k]) for k in range(3))
                first = np.concatenate(
                    [order[start[b]:start[b + cn[0]]] for b in
                     [((z0 + z) * nc[1] + y0 + y) * nc[0] + x0
                      for z in range(cn[2]) for y in range(cn[1])]])
                if first.size == 0:
                    continue
                js, sh = [], []
                for lz in range(nz_lo, cn[2] + nz_hi + 1):
                    sz, cz = divmod(z0 + lz, nc[2])
                    ylo, yhi = tab["ny"][sz]
                    for ry in range(ylo, cn[1] + yhi + 1):
                        sy, cy = divmod(y0 + ry, nc[1])
                        a, b = row_range(cn, (lz, ry, sz, sy))
                        xlo, xhi = tab["nx"][(sz, sy)]
                        kept += max(0, cn[0] + b - a + 1)
                        whole += cn[0] + xhi - xlo + 1
                        assert a >= xlo and b <= xhi
                        for ux in range(x0 + a, x0 + cn[0] + b + 1):
                            sx, cx = divmod(ux, nc[0])
                            k = (cz * nc[1] + cy) * nc[0] + cx
                            mem = order[start[k]:start[k + 1]]
                            js.append(mem)
                            sh.append(np.repeat((sx * H[0] + sy * H[1] + sz * H[2])[None],
                                                mem.size, 0))
                js, sh = np.concatenate(js), np.concatenate(sh)
                d = wr[first][:, None, :] - (wr[js] + sh)[None, :, :]
                a, b = np.nonzero((d ** 2).sum(-1) < rmax * rmax)
                np.add.at(got, (first[a], js[b]), 1)
    d = ref_image(pos[:, None, :] - pos[None, :, :], np.array(L3), tilt)
    want = (d ** 2).sum(-1) < rmax * rmax
    # pairs within the rounding of rmax may fall on either side here (the
    # kernel decides them in FP64 from the original coordinates)
    sure = np.abs(np.sqrt((d ** 2).sum(-1)) - rmax) > 1e-10
    if faces:
        # an atom half a box away has two images at the same distance
        sure &= (np.abs(np.abs(d) - np.array(L3) / 2) > 1e-9).all(-1)
    assert np.array_equal(got[sure], want.astype(int)[sure])
    assert want.sum() > N
    # the corners of the box of cells are gone (at reach 1 every row touches
    # the block: nothing to trim but what tilted images leave)
    assert kept < whole if m > 1 else kept <= whole
