"""The all-pairs kernel's units (host planner): they cover every pair, and what a
CTA counts between two flushes fits its 32-bit bins at any atom count."""
import pytest

from analisi_gb300 import engine

GROUP, CHUNK, WARPS = 64, 128, 8
ATOMS = [1, 2, 31, 64, 65, 127, 128, 129, 300, 1000, 5003, 16384, 131072, 1 << 20,
         4194175, 4194176, 4194177, (1 << 22) + 1, (1 << 23) - 1, 1 << 23, (1 << 23) + 1,
         (1 << 24) + 5, 100_000_000, (1 << 30) - 1]


@pytest.mark.parametrize("natoms,nparts", [(n, k) for n in ATOMS for k in (1, 3, 8) if k <= n])
@pytest.mark.parametrize("frames", [1, 7, 2500, 10 ** 6])
def test_units_cover_the_pairs_and_fit_the_bins(built_engine, natoms, nparts, frames):
    u = engine.allpairs_query(natoms, nparts, frames)
    longest = natoms - (nparts - 1) * (natoms // nparts)
    assert 1 <= u["first"] <= GROUP and u["chunks"] >= 1
    assert u["groups"] * u["first"] >= longest > (u["groups"] - 1) * u["first"]
    chunks = -(-natoms // CHUNK)
    assert u["parts"] * u["chunks"] >= chunks > (u["parts"] - 1) * u["chunks"]
    # the end of the last part is a 32-bit index in the kernel
    assert u["parts"] * u["chunks"] * CHUNK < 2 ** 31
    # a CTA starts a chunk of at most `most` units (a unit a warp at least) with at
    # most 2^31 - 1 pairs counted
    unit = u["first"] * min(natoms, u["chunks"] * CHUNK)
    assert max(u["most"], WARPS) * unit <= 2 ** 31
