"""Bin thresholds found from a guess, on the CPU: each is the first FP64 squared
distance whose bin under the reference's arithmetic (floorf of the float
quotient, lib/src/gofrt.cpp:110) is at least the bin's number, whatever the
guess was worth."""
import numpy as np
import pytest

from analisi_gb300 import engine


@pytest.mark.parametrize("rmin,rmax,nbin", [
    (0.0, 5.5, 80), (0.7, 3.5, 200), (0.0, 1.0, 1), (-2.0, 3.0, 50), (-3.0, 2.0, 7),
    (1e-300, 1e-299, 5), (0.0, 1e150, 40), (1e8, 1e8 + 1e-3, 30), (4.0, 4.0 + 4e-15, 9),
    (0.0, 12.0, 100003)])
def test_thresholds_are_the_first_value_of_their_bin(built_engine, rmin, rmax, nbin):
    th = engine.bin_thresholds(rmin, rmax, nbin)
    dr = (rmax - rmin) / nbin

    def raw(x):
        with np.errstate(over="ignore"):
            return np.floor(np.float32((np.sqrt(x) - rmin) / dr))

    if not th.any():  # nothing can be counted
        x = np.linspace(rmin * rmin, rmax * rmax, 1001)
        r = raw(x)
        assert not ((r >= 0) & (r < nbin)).any()
        return
    end = th[nbin]
    b = np.arange(1, nbin)
    inner = b[(th[b] > th[0]) & (th[b] < end)]
    assert (raw(th[inner]) >= inner).all()
    assert (raw(np.nextafter(th[inner], 0.0)) < inner).all()
    at0 = b[th[b] == th[0]]
    assert (raw(th[at0]) >= at0).all()
    past = b[th[b] == end]
    assert (raw(np.nextafter(end, 0.0)) < past).all()
    assert raw(th[0]) >= 0 and th[0] >= rmin * rmin
    assert th[0] == rmin * rmin or raw(np.nextafter(th[0], 0.0)) < 0
    last = np.nextafter(end, 0.0)
    assert raw(last) < nbin and last <= rmax * rmax
    assert last == rmax * rmax or raw(end) >= nbin
    assert (np.diff(th) >= 0).all()
