"""The work that users of analisi_gb300 have it do, as cases that can be timed.

A case names an entry point (`kind`) and its sizes.  Inputs are random walks of
atoms in a periodic box (and, for `lattice` starts, a thermally disordered
crystal, whose distances crowd into few bins), made from the seed alone.  The
frames are resident before a pass starts, as they are in a program that runs
several calculations on one trajectory; results come back to the host in every
pass.
"""
import math

import numpy as np
import torch

import analisi_gb300
from analisi_gb300 import engine

_SPHERE = 4.18879020478639


def listed():
    return [
        # a few hundred atoms, six lags: a unit-cell study, or one step of a parameter
        # scan; latency of one call
        dict(name="gofr_tiny_300", kind="gofr", natoms=300, ntypes=3, density=0.1736, rmax=5.5,
             rmin=0.0, nbin=80, sigma=0.15, lattice=False, tric=False, npt=False, tmax=6, skip=3,
             every=1, origins=6),
        # 1000 atoms, first coordination shell only, 20 lags: the usual small run
        dict(name="gofr_small_1000", kind="gofr", natoms=1000, ntypes=2, density=0.09391, rmax=3.5,
             rmin=0.7, nbin=200, sigma=0.05, lattice=False, tric=False, npt=False, tmax=20,
             skip=10, every=1, origins=18),
        # a couple of thousand atoms out to almost half the box: g(r,t) of a dense system
        # of ordinary size, half of all pairs counted
        dict(name="gofr_dense_2187", kind="gofr", natoms=2187, ntypes=3, density=0.1, rmax=13.5,
             rmin=0.0, nbin=300, sigma=0.06, lattice=True, tric=False, npt=False, tmax=50, skip=5,
             every=1, origins=40),
        # 16k atoms, one dominant and two trace species, to 12 A: the headline workload,
        # 25 origins by 100 lags
        dict(name="gofr_16k", kind="gofr", natoms=16384, ntypes=3, density=0.1, rmax=12.0,
             rmin=0.0, nbin=400, sigma=0.08, lattice=False, tric=False, npt=False, tmax=100,
             skip=4, every=1, origins=25),
        # a sheared (triclinic) cell, 32k atoms, wrapped coordinates, to 15 A
        dict(name="gofr_tric_32k", kind="gofr", natoms=32768, ntypes=2, density=0.09553, rmax=15.0,
             rmin=0.0, nbin=500, sigma=0.1, lattice=False, tric=True, npt=False, tmax=20, skip=5,
             every=1, origins=10),
        # the largest systems: 131k atoms of four species to 10 A
        dict(name="gofr_131k", kind="gofr", natoms=131072, ntypes=4, density=0.1, rmax=10.0,
             rmin=0.0, nbin=250, sigma=0.1, lattice=False, tric=False, npt=False, tmax=10, skip=10,
             every=1, origins=5),
        # the drop-in pyanalisi.Gofrt as scripts written for the reference call it, with
        # four threads asked for: the result is the exact fold of four partitions
        dict(name="dropin_threads_5488", kind="dropin", natoms=5488, ntypes=3, density=0.1,
             rmax=9.0, rmin=0.0, nbin=300, sigma=0.08, lattice=True, tric=False, npt=False,
             tmax=40, skip=5, every=1, origins=20, nthreads=4),
        # g(r,t) per segment of a constant-pressure run (another box in every frame),
        # normalised by the shell volumes on the GPU
        dict(name="segments_npt_4999", kind="segments", natoms=4999, ntypes=2, density=0.1,
             rmax=10.0, rmin=0.0, nbin=250, sigma=0.08, lattice=False, tric=False, npt=True,
             tmax=20, skip=5, every=1, origins=5, segments=4),
        # many uneven trajectories (parameter sweeps, replicas) in one captured launch
        dict(name="batch_uneven_12", kind="batch", members=12, nmin=256, nmax=16384, rmax=10.0,
             nbin=300, tmax=25, origins=10),
        # mean square displacement of three species, 100 origins by 100 lags
        dict(name="msd_16k", kind="msd", natoms=16384, ntypes=3, density=0.1, sigma=0.08,
             tmax=100, skip=2, origins=100, centres=False),
        # the same with both centre-of-mass options, an odd size, three even species
        dict(name="msd_centres_5003", kind="msd", natoms=5003, ntypes=3, density=0.1, sigma=0.08,
             tmax=80, skip=3, origins=60, centres=True),
        # neighbour lists of one frame, sorted by distance, for coordination analysis
        dict(name="neigh_16k", kind="neigh", natoms=16384, ntypes=3, density=0.1, cutoff=3.5,
             sort=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gofr", "gofr", "gofr", "gofr", "dropin", "segments", "batch", "msd", "msd",
                       "neigh"])
    if kind == "batch":
        return dict(kind="batch", members=rng.randint(4, 16), nmin=256, nmax=_log(rng, 2000, 16384),
                    rmax=round(rng.uniform(6.0, 10.0), 2), nbin=rng.randint(100, 400),
                    tmax=rng.randint(5, 25), origins=rng.randint(3, 10))
    if kind == "msd":
        n = _log(rng, 1000, 16384)
        return dict(kind="msd", natoms=n, ntypes=rng.randint(1, 4), density=0.1,
                    sigma=round(rng.uniform(0.02, 0.15), 3), tmax=rng.randint(10, 100),
                    skip=rng.randint(1, 5), origins=rng.randint(10, 100),
                    centres=rng.random() < 0.4)
    if kind == "neigh":
        return dict(kind="neigh", natoms=_log(rng, 1500, 16384), ntypes=rng.randint(1, 4),
                    density=round(rng.uniform(0.05, 0.1), 4),
                    cutoff=round(rng.uniform(2.6, 3.5), 2), sort=rng.random() < 0.7)
    density = round(rng.uniform(0.05, 0.12), 4)
    n = _log(rng, 300, 131072) if kind == "gofr" else _log(rng, 1000, 16384)
    tric = kind == "gofr" and rng.random() < 0.25
    box = (n / density) ** (1.0 / 3.0)
    # up to the half box for small systems, to 15 A for large ones
    rmax = round(min(rng.uniform(3.5, 15.0), 0.48 * box), 2)
    tmax, origins = rng.randint(5, 60), rng.randint(3, 40)
    npt = kind in ("gofr", "segments") and rng.random() < 0.25
    # no more than the largest listed case: a constant box and one thread let far pairs be
    # skipped, else every pair may have to be looked at
    reach = min(1.0, (2.6 * rmax / box) ** 3) if kind == "gofr" and not npt else 1.0
    most = 6e10 / (reach * n * n)
    while tmax * origins > max(most, 6) and (tmax > 2 or origins > 2):
        tmax, origins = max(2, tmax * 2 // 3), max(2, origins * 2 // 3)
    c = dict(kind=kind, natoms=n, ntypes=rng.randint(1, 4), density=density, rmax=rmax,
             rmin=rng.choice([0.0, 0.0, 0.7]), nbin=rng.randint(80, 500),
             sigma=round(rng.uniform(0.02, 0.15), 3), lattice=rng.random() < 0.4 and not tric,
             tric=tric, npt=npt, tmax=tmax,
             skip=rng.randint(2, 8), every=rng.choice([1, 1, 2]), origins=origins)
    if kind == "dropin":
        c["nthreads"] = rng.choice([1, 2, 4, 8])
        c["every"] = 1
    if kind == "segments":
        c["segments"] = rng.randint(2, 5)
        c["origins"] = max(2, c["origins"] // c["segments"])
        c["every"] = 1
    return c


# --- inputs ------------------------------------------------------------------------------


def _type_ids(n, ntypes, rng, trace=False):
    """Dense ids of every type, shuffled over the atoms; trace: one dominant species."""
    if trace and ntypes > 1:
        few = max(1, n // 1024)
        counts = [n - few * (ntypes - 1)] + [few] * (ntypes - 1)
    else:
        counts = [n // ntypes] * ntypes
        counts[0] += n - sum(counts)
    ids = np.repeat(np.arange(ntypes, dtype=np.int32), counts)
    rng.shuffle(ids)
    return ids


def _frames(n, nframes, L, sigma, lattice, tric, npt, seed):
    """positions [T][N][3] and boxes [T][6 or 9] (internal format), float64 host arrays."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7fffffff)
    kw = dict(generator=g, device="cuda", dtype=torch.float64)
    if lattice:
        side = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
        k = torch.arange(n, device="cuda")
        cell = torch.stack([k % side, (k // side) % side, k // (side * side)], dim=1).double()
        first = (cell + 0.5) / side + torch.randn((n, 3), **kw) * (0.12 / side)
    else:
        first = torch.rand((n, 3), **kw)
    tilt = (0.3 * L, 0.2 * L, 0.1 * L) if tric else (0.0, 0.0, 0.0)
    h = torch.tensor([[L, tilt[0], tilt[1]], [0.0, L, tilt[2]], [0.0, 0.0, L]],
                     dtype=torch.float64, device="cuda")
    pos = torch.randn((nframes, n, 3), **kw)
    pos *= sigma
    pos[0] = first @ h.T
    pos = torch.cumsum(pos, dim=0)
    if tric:  # wrapped into the cell, frame by frame
        frac = pos @ torch.linalg.inv(h).T
        pos = (frac - torch.floor(frac)) @ h.T
    box = np.zeros((nframes, 9 if tric else 6))
    scale = np.ones(nframes)
    if npt:
        r = np.random.default_rng(seed)
        scale = 1.0 + 0.004 * np.cumsum(r.normal(size=nframes)) / math.sqrt(nframes) \
            + 0.001 * r.normal(size=nframes)
        pos *= torch.from_numpy(scale).cuda()[:, None, None]
    box[:, 3:6] = (0.5 * L * scale)[:, None]
    if tric:
        box[:, 6:9] = np.array(tilt)[None, :] * scale[:, None]
    return pos.cpu().numpy(), box


def _steps(c):
    """(ntimesteps, frames) of a case: lags 0 .. tmax-1 need ntimesteps >= tmax."""
    n = max(c["origins"] * c["skip"], c["tmax"])
    return n, n + c["tmax"]


def _edge(c):
    return (c["natoms"] / c["density"]) ** (1.0 / 3.0)


def _gofr_inputs(c, seed, frames):
    rng = np.random.default_rng(seed)
    pos, box = _frames(c["natoms"], frames, _edge(c), c["sigma"], c["lattice"], c["tric"],
                       c["npt"], seed)
    trace = c["natoms"] > 10000 and c["ntypes"] == 3
    return pos, box, _type_ids(c["natoms"], c["ntypes"], rng, trace)


def _members(c, seed):
    """Trajectories of a batch: the sizes belong to the case, the coordinates to the seed."""
    r = np.random.default_rng(1000 + c["members"])
    out = []
    for k in range(c["members"]):
        lo, hi = math.log(c["nmin"]), math.log(c["nmax"])
        n = int(round(math.exp(lo + (hi - lo) * (k + r.uniform()) / c["members"])))
        nt = int(r.integers(1, 5))
        out.append(dict(natoms=n, ntypes=nt, sigma=float(r.uniform(0.02, 0.15)),
                        skip=int(r.integers(3, 8)), seed=int(seed) * 131 + k))
    return out


def _member_case(c, m):
    return dict(natoms=m["natoms"], ntypes=m["ntypes"], density=0.1, rmax=c["rmax"], rmin=0.0,
                nbin=c["nbin"], sigma=m["sigma"], lattice=False, tric=False, npt=False,
                tmax=c["tmax"], skip=m["skip"], every=1, origins=c["origins"])


def _windows(c):
    n, _ = _steps(c)
    return [k * n for k in range(c["segments"])]


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        trajs = []
        for m in _members(c, seed):
            mc = _member_case(c, m)
            n, frames = _steps(mc)
            pos, box, ids = _gofr_inputs(mc, m["seed"], frames)
            trajs.append(dict(positions=pos, boxes=box, type_ids=ids, ntypes=m["ntypes"],
                              params=engine.make_params(0.0, c["rmax"], c["nbin"], c["tmax"],
                                                        m["skip"], 1, n, 0)))
        e = engine.Engine(0)
        e.batch_set(trajs)
        return dict(case=c, engine=e, out=np.zeros(e._batch[1], dtype=np.uint64))
    if c["kind"] == "dropin":
        pa = analisi_gb300.load_pyanalisi()
        n, frames = _steps(c)
        pos, box, ids = _gofr_inputs(c, seed, frames)
        lammps = np.zeros((frames, 6))
        lammps[:, 1::2] = 2.0 * box[:, 3:6]
        traj = pa.Trajectory(pos, np.zeros_like(pos), ids, lammps, pa.BoxFormat.LammpsOrtho, False,
                             False)
        g = pa.Gofrt(traj, c["rmin"], c["rmax"], c["nbin"], c["tmax"], c["nthreads"], c["skip"],
                     c["every"], False)
        return dict(case=c, traj=traj, gofrt=g, n=n)
    e = engine.Engine(0)
    state = dict(case=c, engine=e)
    if c["kind"] in ("gofr", "segments"):
        n, frames = _steps(c)
        state["n"] = n
        total = frames if c["kind"] == "gofr" else _windows(c)[-1] + frames
        pos, box, ids = _gofr_inputs(c, seed, total)
        if c["kind"] == "gofr":
            leff = min(c["tmax"], n)
            state["out"] = np.zeros(leff * c["ntypes"] * (c["ntypes"] + 1) * c["nbin"],
                                    dtype=np.uint64)
    elif c["kind"] == "msd":
        frames = max(c["origins"] * c["skip"], c["tmax"]) + c["tmax"]
        pos, box = _frames(c["natoms"], frames, _edge(c), c["sigma"], False, False, False, seed)
        ids = _type_ids(c["natoms"], c["ntypes"], np.random.default_rng(seed))
    else:
        pos, box = _frames(c["natoms"], 3, _edge(c), 0.08, False, False, False, seed)
        ids = _type_ids(c["natoms"], c["ntypes"], np.random.default_rng(seed))
        # room for the densest neighbourhood of a random gas
        mean = c["density"] * _SPHERE * c["cutoff"] ** 3 / c["ntypes"]
        room = int(mean + 9.0 * math.sqrt(mean) + 8)
        state["spec"] = [(room, c["cutoff"] ** 2, 0.0)] * c["ntypes"]
    e.set_frames(pos, box, ids, c["ntypes"])
    if c.get("centres"):
        e.set_centres(_centres(pos, ids, c["ntypes"]))
    return state


def _centres(pos, ids, ntypes):
    return np.stack([pos[:, ids == k].mean(axis=1) for k in range(ntypes)], axis=1)


# --- one pass ----------------------------------------------------------------------------


def run(state):
    c = state["case"]
    if c["kind"] == "dropin":
        g = state["gofrt"]
        g.reset(state["n"])
        g.calculate(0)
        return np.array(g, copy=True)
    e = state["engine"]
    if c["kind"] == "gofr":
        return e.run(c["rmin"], c["rmax"], c["nbin"], c["tmax"], c["skip"], c["every"],
                     state["n"], 0, out=state["out"])
    if c["kind"] == "segments":
        out, _ = e.gofr(c["rmin"], c["rmax"], c["nbin"], c["tmax"], c["skip"], c["every"],
                        state["n"], _windows(c), norm="shell")
        return out
    if c["kind"] == "batch":
        return e.batch_run(use_graph=True, out=state["out"])
    if c["kind"] == "msd":
        return e.msd(c["skip"], c["tmax"], max(c["origins"] * c["skip"], c["tmax"]), 0,
                     c["centres"], c["centres"])
    lists = e.neighbours(1, state["spec"], c["sort"])
    return [lists.list, lists.rpos]


# --- what a pass cannot do without -------------------------------------------------------


def _gofr_work(c, windows=1, out_item=8):
    """Coordinates of every frame once, the counts once; three differences, their squares, a
    root, a scaling and a rounding for each pair within rmax."""
    n, frames = _steps(c)
    lags = -(-min(c["tmax"], n) // c["every"])
    N = c["natoms"]
    inside = min(1.0, _SPHERE * c["rmax"] ** 3 / _edge(c) ** 3)
    items = float(windows) * lags * -(-n // c["skip"])
    outs = windows * min(c["tmax"], n) * c["ntypes"] * (c["ntypes"] + 1) * c["nbin"] * out_item
    return {"bytes": (n * (windows - 1) + frames) * N * 24.0 + outs,
            "flops": items * N * N * inside * 11.0}


def work(case):
    c = case
    if c["kind"] in ("gofr", "dropin"):
        return _gofr_work(c)
    if c["kind"] == "segments":
        return _gofr_work(c, c["segments"])
    if c["kind"] == "batch":
        w = [_gofr_work(_member_case(c, m)) for m in _members(c, 0)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    if c["kind"] == "msd":
        n = max(c["origins"] * c["skip"], c["tmax"])
        items = float(c["tmax"]) * -(-n // c["skip"])
        return {"bytes": (n + c["tmax"]) * c["natoms"] * 24.0,
                "flops": items * c["natoms"] * (11.0 if c["centres"] else 8.0)}
    near = c["density"] * _SPHERE * c["cutoff"] ** 3
    return {"bytes": c["natoms"] * (24.0 + near * 40.0), "flops": c["natoms"] * near * 9.0}


# --- the same in 64 bits, without the package --------------------------------------------


def _minimum_image(d, box):
    """z, then y, then x, one edge at a time (the tilts go with the edge)."""
    tric = len(box) == 9
    for ax in (2, 1, 0):
        half = float(box[3 + ax])
        while True:
            s = (d[ax] > half).double() - (d[ax] < -half).double()
            if not bool((s != 0).any()):
                break
            d[ax] = d[ax] - s * (2.0 * half)
            if tric and ax == 2:
                d[1] = d[1] - s * float(box[8])
                d[0] = d[0] - s * float(box[7])
            if tric and ax == 1:
                d[0] = d[0] - s * float(box[6])
    return d


def _counts(pos, boxes, ids, ntypes, c, n, primo, parts):
    """Counts [parts][leff][channel][bin], partitions of the first atoms by index."""
    N, nbin = c["natoms"], c["nbin"]
    half = ntypes * (ntypes + 1) // 2
    lo = torch.minimum(ids[:, None], ids[None, :])
    hi = torch.maximum(ids[:, None], ids[None, :])
    channel = half - (hi + 1) * (hi + 2) // 2 + lo
    eye = torch.arange(N, device="cuda")
    channel[eye, eye] += half
    leff = min(c["tmax"], n)
    dr = (c["rmax"] - c["rmin"]) / nbin
    out = torch.zeros((parts, leff, 2 * half * nbin), dtype=torch.int64, device="cuda")
    per = N // parts
    rows = max(1, min(N, 40_000_000 // N))
    for o in range(primo, primo + n, c["skip"]):
        for lag in range(0, leff, c["every"]):
            for q in range(parts):
                end = N if q == parts - 1 else (q + 1) * per
                for a in range(q * per, end, rows):
                    b = min(a + rows, end)
                    d = [pos[o, a:b, k, None] - pos[o + lag, None, :, k] for k in range(3)]
                    d = _minimum_image(d, boxes[o])
                    d2 = d[0] * d[0]
                    d2 = d2 + d[1] * d[1]
                    d2 = d2 + d[2] * d[2]
                    f = torch.floor(((torch.sqrt(d2) - c["rmin"]) / dr).float())
                    ok = (d2 <= c["rmax"] * c["rmax"]) & (d2 >= c["rmin"] * c["rmin"]) & \
                        (f >= 0) & (f < nbin)
                    at = channel[a:b][ok] * nbin + f[ok].long()
                    out[q, lag] += torch.bincount(at, minlength=2 * half * nbin)
    return out.reshape(parts, leff, 2 * half, nbin)


def _gofr_exact(c, seed, parts, windows):
    n, frames = _steps(c)
    N = c["natoms"]
    items = len(windows) * -(-min(c["tmax"], n) // c["every"]) * -(-n // c["skip"])
    if items * float(N) * N > 4e10 or items * parts > 12000:
        return None
    pos, box, ids = _gofr_inputs(c, seed, windows[-1] + frames)
    pos, ids = torch.from_numpy(pos).cuda(), torch.from_numpy(ids).cuda().long()
    return [_counts(pos, box, ids, c["ntypes"], c, n, w, parts) for w in windows], n


def exact(case, seed):
    c = case
    if c["kind"] == "gofr":
        got = _gofr_exact(c, seed, 1, [0])
        return None if got is None else got[0][0][0].cpu().numpy().astype(np.uint64)
    if c["kind"] == "dropin":
        got = _gofr_exact(c, seed, c["nthreads"], [0])
        return None if got is None else (got[0][0].sum(0).double() / (got[1] // c["skip"])).cpu()
    if c["kind"] == "segments":
        got = _gofr_exact(c, seed, 1, _windows(c))
        if got is None:
            return None
        dr = (c["rmax"] - c["rmin"]) / c["nbin"]
        r = np.arange(c["nbin"] + 1) * dr + c["rmin"]
        shell = 4.0 * math.pi / 3.0 * (r[1:] ** 3 - r[:-1] ** 3)
        return np.stack([(w[0].double() / (got[1] // c["skip"])).cpu().numpy() / shell
                         for w in got[0]])
    if c["kind"] == "msd":
        return _msd_exact(c, seed)
    if c["kind"] == "neigh":
        return _neigh_exact(c, seed)
    return None


def _msd_exact(c, seed):
    n = max(c["origins"] * c["skip"], c["tmax"])
    pos, _ = _frames(c["natoms"], n + c["tmax"], _edge(c), c["sigma"], False, False, False, seed)
    ids = _type_ids(c["natoms"], c["ntypes"], np.random.default_rng(seed))
    cm = torch.from_numpy(_centres(pos, ids, c["ntypes"])).cuda()
    by = [torch.from_numpy(pos[:, ids == k]).cuda() for k in range(c["ntypes"])]
    out = torch.zeros((c["tmax"], 2 if c["centres"] else 1, c["ntypes"]), dtype=torch.float64,
                      device="cuda")
    o = torch.arange(0, n, c["skip"], device="cuda")
    for lag in range(c["tmax"]):
        dc = cm[o] - cm[o + lag]
        for k in range(c["ntypes"]):
            s = torch.zeros((), dtype=torch.float64, device="cuda")
            for part in torch.split(torch.arange(len(o), device="cuda"), 32):
                d = by[k][o[part]] - by[k][o[part] + lag]
                if c["centres"]:
                    d = d - dc[part, k][:, None, :]
                s = s + (d * d).sum()
            out[lag, 0, k] = s / (len(o) * by[k].shape[1])
        if c["centres"]:
            out[lag, 1] = (dc * dc).sum(2).mean(0)
    return out.cpu().numpy()


def _neigh_exact(c, seed):
    N, nt = c["natoms"], c["ntypes"]
    pos, box = _frames(N, 3, _edge(c), 0.08, False, False, False, seed)
    ids = _type_ids(N, nt, np.random.default_rng(seed))
    mean = c["density"] * _SPHERE * c["cutoff"] ** 3 / nt
    room = int(mean + 9.0 * math.sqrt(mean) + 8)
    x = torch.from_numpy(pos[1]).cuda()
    lists = np.zeros((nt, N, room + 1), dtype=np.uint64)
    rpos = np.zeros((nt, N, room, 4))
    rows = max(1, 40_000_000 // N)
    for a in range(0, N, rows):
        b = min(a + rows, N)
        d = _minimum_image([x[a:b, k, None] - x[None, :, k] for k in range(3)], box[1])
        d2 = d[0] * d[0]
        d2 = d2 + d[1] * d[1]
        d2 = d2 + d[2] * d[2]
        near = d2 <= c["cutoff"] ** 2
        i = torch.arange(a, b, device="cuda")
        near[i - a, i] = False
        at = torch.nonzero(near)
        v = torch.stack([torch.sqrt(d2[near]), d[0][near], d[1][near], d[2][near]], 1).cpu().numpy()
        i, j = at[:, 0].cpu().numpy() + a, at[:, 1].cpu().numpy()
        order = np.lexsort((j, v[:, 0], i)) if c["sort"] else np.lexsort((j, i))
        i, j, v = i[order], j[order], v[order]
        for k in range(nt):
            of = ids[j] == k
            ik, jk, vk = i[of], j[of], v[of]
            first = np.searchsorted(ik, ik)
            slot = np.arange(len(ik)) - first
            lists[k, ik, 1 + slot] = jk
            lists[k, :, 0] += np.bincount(ik, minlength=N).astype(np.uint64)
            rpos[k, ik, slot] = vk
    return [lists.reshape(-1), rpos.reshape(-1)]
