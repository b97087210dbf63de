"""A streamed run keeps to its device budget with the cell lists it builds: with
little more than the budget to be had (ANALISI_GB300_MAX_ALLOC) it takes the same
path as with all of the memory, instead of falling back to all pairs."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import json, os, sys
import numpy as np
sys.path.insert(0, {root!r})
from analisi_gb300 import engine
N, T, L, tric = 20000, 460, (20000 / 0.1) ** (1.0 / 3.0), {tric}
rng = np.random.default_rng(1)
step = rng.normal(0.0, 0.05, (20, N, 3))
start = rng.uniform(0.0, L, (1, N, 3))
pos = np.ascontiguousarray(np.broadcast_to(start, (T, N, 3)))
for f in range(T):
    pos[f] += step[f % 20]
box = np.zeros((T, 9 if tric else 6))
box[:, 3:6] = L / 2
if tric:
    box[:, 6:] = [0.2 * L, 0.1 * L, 0.1 * L]
ids = (np.arange(N) % 2).astype(np.int32)
out = []
with engine.Engine(0) as e:
    # the first run of each path loads its kernels; 3 frames stay resident after it
    for n, kernel in ((1, "f32"), (1, "auto"), (450, "auto"), (450, "auto")):
        if len(out) == 3:
            os.environ["ANALISI_GB300_MAX_ALLOC"] = str({budget} // 1000000 + 16)
        e.set_frames(pos[:3], box[:3], ids, 2)
        before = e.stats()["launches"]
        c = e.run_streamed(pos, box, ids, 2, {budget}, 0.0, {rmax}, 100, 2, 10, 1, n, 0,
                           kernel=kernel)
        out.append([e.stats()["launches"] - before, c.sum(axis=(0, 1)).tolist()])
print(json.dumps(out[2:]))
"""

BUDGET = 400_000_000  # bytes: 312 of the 460 frames


@pytest.mark.parametrize("rmax", [3.3, 3.6, 8.0])
@pytest.mark.parametrize("tric", [False, True])
def test_cell_lists_fit_the_budget(built_engine, rmax, tric):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=root, budget=BUDGET, rmax=rmax,
                                                           tric=tric)],
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr
    free, limited = json.loads(p.stdout.strip().splitlines()[-1])
    assert free == limited
