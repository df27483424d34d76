"""The serving scheduler under a mix of requests that stay resident (large ones)
and requests that run in joint calls (small ones): neither holds up the other
for long, closing waits for one call at most, and records equal cz_census's."""
import time

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def tup(recs):
    return [(r.p, [(v.r, v.M, v.L, v.witness, v.K) for v in r.profiles], r.a4) for r in recs]


@pytest.fixture(scope="module")
def alone():
    from rabung_atlas32_b200.census import Census
    with Census() as c:
        yield lambda primes: tup(c.profiles(primes, mode="auto", a4=True))


def order_of(srv, n):
    """Request ids in the order in which they complete."""
    done = []
    while len(done) < n:
        rid = srv.next_done(60000)
        assert rid is not None
        done.append(rid)
    return done


def test_close_waits_for_one_call_at_most():
    """Some four seconds of small requests are waiting when the server closes."""
    from rabung_atlas32_b200.serving import Server
    srv = Server(slots=1, slot_budget_mb=1024)
    for k in range(400):
        srv.submit(4200000000 + 100000 * (k % 50), 100)
    time.sleep(0.3)
    t0 = time.perf_counter()
    srv.close()
    assert time.perf_counter() - t0 < 2.0


def test_resident_request_keeps_its_share(alone):
    """A request of some 0.1 s of filter time, then over a second of small ones:
    it ends well before they do."""
    from rabung_atlas32_b200.serving import Server
    srv = Server(slots=1, slot_budget_mb=4096)
    try:
        big = srv.submit(4280000000, 512)
        small = [srv.submit(4100000000 + 100000 * k, 100) for k in range(120)]
        order = order_of(srv, 121)
        assert order.index(big) < 70
        primes, recs = srv.fetch(big, 512)
        assert primes == sieve.primes_from(4280000000, 512) and tup(recs) == alone(primes)
        for rid in (small[0], small[-1]):
            primes, recs = srv.fetch(rid, 100)
            assert tup(recs) == alone(primes)
    finally:
        srv.close()


def test_small_request_passes_one_that_waits_for_space(alone):
    """Two large requests of which the planes of one fit: a small one that
    arrives while the second waits is answered before the first ends."""
    from rabung_atlas32_b200.serving import Server
    srv = Server(slots=1, slot_budget_mb=3072)
    try:
        first, second = srv.submit(4280000000, 1200), srv.submit(4270000000, 1200)
        time.sleep(0.06)
        small = srv.submit(4000000007, 4)
        order = order_of(srv, 3)
        assert order == [small, first, second]
        for rid, n in ((small, 4), (second, 1200)):
            primes, recs = srv.fetch(rid, n)
            assert tup(recs) == alone(primes)
    finally:
        srv.close()


def test_counters_of_a_joint_call_that_is_refused(alone):
    """Three requests meet in one call; one asks for the sparse route below its
    reach and is refused, the others' speculative misses (margin 0) are counted."""
    import dataclasses
    from rabung_atlas32_b200 import _lib
    from rabung_atlas32_b200.census import Census, CensusError, Tuning
    from rabung_atlas32_b200.serving import Server
    with Census() as probe:
        tuning = dataclasses.replace(probe.tuning, spec_margin10=(0,) * 10)
    assert isinstance(tuning, Tuning)
    srv = Server(slots=1, slot_budget_mb=1024, tuning=tuning)
    flags = _lib.CZ_SPARSE | _lib.CZ_A4
    try:
        srv.submit(4200000000, 100, flags | _lib.CZ_VERIFY)       # keeps the server busy while the three arrive
        goods = [srv.submit(4290000000, 60, flags), srv.submit(4280000000, 30, flags)]
        bad = srv.submit(101, 5, flags)
        for rid, n in zip(goods, (60, 30)):
            primes, recs = srv.fetch(rid, n)
            assert tup(recs) == alone(primes)
        with pytest.raises(CensusError, match="sparse path unsupported"):
            srv.fetch(bad, 5)
        order_of(srv, 1)
        busy = srv.stats()["respec_primes"]
    finally:
        srv.close()
    with Census(tuning=tuning) as c:
        want = 0
        for lo, n in ((4200000000, 100), (4290000000, 60), (4280000000, 30)):
            c.raw(sieve.primes_from(lo, n), mode="sparse", a4=False)
            assert c.last_stats["n_respec"] > 0
            want += c.last_stats["n_respec"]
    assert busy == want
