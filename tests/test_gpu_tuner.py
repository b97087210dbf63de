"""What the tuner measures and where its choices are found again."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu


def _child(case, kernels, env):
    here = os.path.dirname(os.path.abspath(__file__))
    out = subprocess.run([sys.executable, os.path.join(here, "tune_child_args.py"),
                          json.dumps(case), *kernels], env={**os.environ, **env},
                         capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr
    return json.loads(out.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("fill", ["0", "255"])
def test_trials_on_a_new_context_do_the_whole_sample(built_engine, tmp_path, fill):
    """The first calculation of a context is a tuned one, in memory that held
    something else: every trial starts from cleared work counters.  The sample
    has 10 lags x 10 origins x 6000^2 = 3.6e9 ordered pairs, which the all-pairs
    kernel cannot do in less than 0.6 ms (seven FP32 operations a pair, 152 SMs x
    128 lanes x 2.07 GHz)."""
    case = dict(seed=88, counts=[3000, 2000, 1000], frames=40, edge=40.0,
                params=dict(rmin=0.0, rmax=5.0, nbin=50, tmax=10, skip=3, every=1,
                            ntimesteps=30, primo=0))
    log = str(tmp_path / "log.txt")
    tuned, plain = _child(case, ["tuned", "f32"], {"ANALISI_GB300_FILL_ALLOC": fill,
                                                   "ANALISI_GB300_TUNE_LOG": log})
    ms = [float(line.rsplit("ms=", 1)[1]) for line in open(log) if " all-pairs " in line]
    assert len(ms) == 1 and ms[0] > 0.6
    assert all(float(line.rsplit("ms=", 1)[1]) > 0.0 for line in open(log))
    assert {**tuned, "kernel_used": 0} == {**plain, "kernel_used": 0}
