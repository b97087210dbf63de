"""The sum of k additions of 1/n, by runs of equal steps, on the CPU: bit for
bit the additions one by one (numpy's cumsum) for every k up to four million;
beyond, each sum is the one before it plus 1/n in FP64 wherever a run can end
(where the sum enters a binade) and at counts far from there
(lib/src/gofrt.cpp:118)."""
import numpy as np
import pytest

from analisi_gb300 import engine


@pytest.mark.parametrize("n", [1, 2, 3, 5, 7, 10, 40, 49, 999, 4097, 1 << 20, 3_000_001,
                               2**31 - 1])
def test_sums_are_the_sequential_ones(built_engine, n):
    incr = 1.0 / n

    def sums(k):
        return engine.counts_to_buffer(k.astype(np.uint64)[None], n, 1, nparts=1)

    K = 4_000_000
    want = np.concatenate([[0.0], np.cumsum(np.full(K, incr))])
    assert np.array_equal(sums(np.arange(K + 1)), want)
    rng = np.random.default_rng(n)
    # where s(k) ~ k / n passes 2^b (the sum lags by its rounding: found by bisection)
    mids = [int(x) for x in 2.0 ** rng.uniform(22, 56, 60)]
    e0 = int(np.frexp(incr)[1])
    for b in range(e0 + 20, e0 + 54):
        lo, hi = 1, 1 << 58
        while hi - lo > 1:
            m = (lo + hi) // 2
            if sums(np.array([m], dtype=np.uint64))[0] >= 2.0 ** b:
                hi = m
            else:
                lo = m
        mids.append(lo)
    for m in mids:
        k = np.arange(max(0, m - 40), m + 40, dtype=np.uint64)
        s = sums(k)
        assert np.array_equal(s[1:], s[:-1] + incr)


def test_partitions_fold_in_order(built_engine):
    rng = np.random.default_rng(5)
    c = rng.integers(0, 1 << 30, (5, 300)).astype(np.uint64)
    each = [engine.counts_to_buffer(c[q:q + 1], 37, 1, nparts=1) for q in range(5)]
    want = each[0]
    for e in each[1:]:
        want = want + e
    assert np.array_equal(engine.counts_to_buffer(c, 37, 1, nparts=5), want)
