"""Both filters, each in calls that reach it: profiles in groups of 32 (calls of
some size) and profiles by themselves (calls of few primes, calls without
speculation, requests resident in a server).  A second library forces what the
default one meets rarely: a group for every profile, small tiles, few warps."""
import contextlib
import dataclasses

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def tup(recs):
    return [(r.p, [(v.r, v.M, v.L, v.witness, v.K) for v in r.profiles]) for r in recs]


def census(ps, mode, tuning=None):
    from rabung_atlas32_b200.census import Census
    with Census(tuning=tuning) as c:
        return tup(c.profiles(ps, mode=mode, a4=False)), c.last_stats


@pytest.fixture(scope="module")
def tuned():
    from rabung_atlas32_b200.census import Census
    with Census() as c:
        return c.tuning


@pytest.fixture(scope="module")
def variant(tmp_path_factory):
    from rabung_atlas32_b200 import _lib, build
    so = tmp_path_factory.mktemp("variant") / "librabung_census_small.so"
    build.compile_library(so, extra=["-DCZ_TILE_WORDS=4096", "-DCZ_GROUP_TILE_WORDS=8192", "-DCZ_GROUP_WARPS=6",
                                     "-DCZ_GROUP_OWN_COST=1e9"])
    lib = _lib.load(so)

    @contextlib.contextmanager
    def use():
        saved = _lib._lib
        _lib._lib = lib
        try:
            yield
        finally:
            _lib._lib = saved
    return use


@pytest.mark.parametrize("count", [31, 32, 33, 64])
@pytest.mark.parametrize("lo", [6_000_011, 16_777_259, 268_435_459])
def test_groups_formed_by_cost(lo, count, tuned):
    ps = sieve.primes_from(lo, count)
    got, st = census(ps, "sparse", tuned)
    # a call without groups takes at most 5 launches, and as many for re-runs
    assert st["kernels"] > 5 + 5 * (st["n_respec"] > 0) and st["n_fallback"] == 0
    assert got == census(ps, "dense")[0]


@pytest.mark.parametrize("lo,count", [(16_384, 64), (70_001, 33), (1 << 20, 1), (1 << 20, 31), (1 << 20, 32),
                                      (1 << 20, 33), (5_000_011, 64), (24_000_001, 65), (268_435_459, 40)])
def test_forced_groups_in_small_tiles(lo, count, tuned, variant):
    """Every profile in a group, from the smallest sparse prime up: all rows
    narrow, or wide chunks of 32 to 64 indices."""
    ps = sieve.primes_from(lo, count)
    with variant():
        got, st = census(ps, "sparse", tuned)
    assert st["n_fallback"] == 0
    assert got == census(ps, "dense")[0]


# calls whose profiles are filtered by themselves: no speculation, or too few primes for a group
def own_calls():
    return [(0, sieve.primes_ending(4294967291, 24) + sieve.primes_from(1 << 24, 24)), (1, sieve.primes_ending(4294967291, 2)),
            (1, [sieve.primes_from(1 << k, 1)[0] for k in range(21, 32)])]


@pytest.mark.parametrize("change", [dict(anchor_t=(0, 0, 2, 2, 2, 2, 2, 2, 2, 2)), dict(anchor_t=(0, 0, 16, 10, 9, 8, 7, 7, 6, 6)),
                                    dict(anchor_t=(0,) * 10), dict(epoch_rows=1), dict(epoch_rows=7), dict(epoch_rows=64),
                                    dict(epoch_rows=1 << 20), dict(cta_per_profile=3), dict(screen=0)])
def test_per_profile_settings_do_not_change_records(change, tuned):
    for speculate, ps in own_calls():
        t = dataclasses.replace(tuned, speculate=speculate)
        want, st = census(ps, "sparse", t)
        assert st["kernels"] <= 5 + 5 * (st["n_respec"] > 0)
        assert census(ps, "sparse", dataclasses.replace(t, **change))[0] == want, (change, speculate, len(ps))


def test_per_profile_small_tiles(tuned, variant):
    ps = sieve.primes_from(1 << 26, 40) + sieve.primes_from(1 << 28, 40) + sieve.primes_ending(1 << 30, 24)
    with variant():
        got, st = census(ps, "sparse", dataclasses.replace(tuned, speculate=0))
    assert st["n_fallback"] == 0 and st["kernels"] <= 5
    assert got == census(ps, "sparse", tuned)[0]


def test_resident_requests_join_and_miss(tuned):
    """Requests above the joint calls' size, the second while the first is being
    filtered: the launch yields, both stay resident, and with margin 0 many
    speculations miss and are run again."""
    import time
    from rabung_atlas32_b200.census import Census
    from rabung_atlas32_b200.serving import Server
    t = dataclasses.replace(tuned, spec_margin10=(0,) * 10)
    reqs = [(4_290_000_000, 768), (4_280_000_000, 256)]
    srv = Server(slots=1, slot_budget_mb=8192, tuning=t)
    try:
        ids = [srv.submit(*reqs[0])]
        time.sleep(0.05)
        ids.append(srv.submit(*reqs[1]))
        got = [srv.fetch(rid, n) for rid, (lo, n) in zip(ids, reqs)]
        st = srv.stats()
    finally:
        srv.close()
    assert st["yields"] >= 1 and st["respec_primes"] > 0 and st["fallback_primes"] == 0
    with Census() as c:
        for (lo, n), (primes, recs) in zip(reqs, got):
            assert primes == sieve.primes_from(lo, n)
            alone = c.profiles(primes, mode="auto", a4=True)
            assert tup(recs) == tup(alone) and [r.a4 for r in recs] == [r.a4 for r in alone]
