"""A loading warp of the grouped filter that gives up on its slot: the item it
holds, the one it had already been handed and the items nobody takes any more
all send their groups to the dense scan, so no record comes from a search that
was cut short."""
import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def tup(recs):
    return [(r.p, [(v.r, v.M, v.L, v.witness, v.K) for v in r.profiles]) for r in recs]


def test_wait_that_runs_out_falls_back(tmp_path):
    """A library whose loading warps wait zero tries for a free slot: each tests
    one item and leaves with the next one in hand."""
    from rabung_atlas32_b200 import _lib, build
    from rabung_atlas32_b200.census import Census, Tuning
    ps = sieve.primes_ending(1 << 28, 64)
    with Census(tuning=Tuning()) as c0:
        want = tup(c0.profiles(ps, mode="dense", a4=False))
    so = tmp_path / "librabung_census_waits.so"
    build.compile_library(so, extra=["-DCZ_GROUP_EMPTY_TRIES=0", "-DCZ_GROUP_FULL_TRIES=500"])
    lib = _lib.load(so)
    saved = _lib._lib
    try:
        _lib._lib = lib
        with Census(tuning=Tuning()) as c1:
            got = c1.profiles(ps, mode="sparse", a4=False)
            assert c1.last_stats["n_fallback"] == len(ps)
            assert tup(got) == want
    finally:
        _lib._lib = saved
