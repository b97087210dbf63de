"""The warp-streamed kernel's u32 bins where a chunk of its units has 2^32 pairs or
more: it adds its histogram to the counts in between.  Same counts as the
all-pairs kernel, whose units are bounded by their size alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 60.0


@pytest.mark.parametrize("nparts", [1, 2])
@pytest.mark.parametrize("heaps", [(6.0, 26.0, 46.0), (6.0, 16.0, 26.0, 36.0, 46.0, 56.0)])
def test_dense_heaps_in_one_chunk(built_engine, nparts, heaps):
    """Heaps of 60000 atoms (3.6e9 pairs each, in a cell or two) ten and twenty
    angstrom apart along x, so that one chunk of units holds several."""
    from analisi_gb300 import engine
    rng = np.random.default_rng(2)
    pos = np.concatenate([[x, 31.0, 31.0] + rng.normal(0.0, 0.3, (60000, 3)) for x in heaps])
    n = len(pos)
    box = np.zeros((1, 6))
    box[0, 3:] = EDGE / 2
    ids = (np.arange(n) % 2).astype(np.int32)
    args = (0.0, 5.0, 100, 1, 1, 1, 1, 0)
    with engine.Engine(0) as e:
        e.set_frames(pos[None], box, ids, 2)
        got = e.run(*args, kernel="auto", nparts=nparts).copy()
        assert e.stats()["kernel_used"] == 5
        want = e.run(*args, kernel="f32", nparts=nparts)
        assert e.stats()["kernel_used"] == 1
    np.testing.assert_array_equal(got, want)
    assert int(got.sum()) > len(heaps) * 3.5e9
