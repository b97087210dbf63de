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


# 3 types x 1500 bins: a histogram the warp-streamed kernel has room for and the
# block cell-list kernel has not
WIDE = dict(seed=91, counts=[2000, 1500, 1000], frames=24, edge=36.0,
            params=dict(rmin=0.0, rmax=4.0, nbin=1500, tmax=8, skip=2, every=1, ntimesteps=16,
                        primo=0))


def test_large_histograms_are_tuned_and_found_again(built_engine, tmp_path):
    """The tuner tries the warp-streamed kernel wherever AUTO takes it, and AUTO
    finds its choice (one changed to the all-pairs kernel shows that it does)."""
    cache, log = str(tmp_path / "cache.txt"), str(tmp_path / "log.txt")
    auto, = _child(WIDE, ["auto"], {})
    tuned, = _child(WIDE, ["tuned"], {"ANALISI_GB300_TUNE_CACHE": cache,
                                      "ANALISI_GB300_TUNE_LOG": log})
    assert auto["kernel_used"] == 5
    assert " warp-cells " in open(log).read() and tuned == auto
    key = open(cache).read().split()[0]
    with open(cache, "w") as f:
        f.write(f"{key} 0 1 4 1 1 1 8 1\n")
    again, = _child(WIDE, ["auto"], {"ANALISI_GB300_TUNE_CACHE": cache})
    assert again == {**auto, "kernel_used": 1}


def test_choices_stored_for_older_kernels_are_not_taken(built_engine, tmp_path):
    """A stored choice compares the kernels of its time: lines whose key starts at
    the job's size, as all did before the key named a version, are left alone."""
    cache = str(tmp_path / "cache.txt")
    tuned, = _child(WIDE, ["tuned"], {"ANALISI_GB300_TUNE_CACHE": cache})
    key = open(cache).read().split()[0]
    with open(cache, "w") as f:
        f.write(f"{key[key.index('n2^'):]} 0 1 4 1 1 1 8 1\n")
    auto, = _child(WIDE, ["auto"], {"ANALISI_GB300_TUNE_CACHE": cache})
    assert auto["kernel_used"] == 5 and auto == tuned
