"""The grouped anchor filter (32 profiles of one order per word) against the
dense scan, bit for bit: group sizes around 32 and the least group, primes from
the smallest sparse one up, so that the filter's rows are all narrow, narrow and
wide, or end inside a row group, and wide ranges of p in one call."""
import time

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    from rabung_atlas32_b200.census import Census
    with Census() as c:
        yield c


def tup(recs):
    return [(r.p, [(v.r, v.M, v.L, v.witness, v.K) for v in r.profiles]) for r in recs]


@pytest.mark.parametrize("lo,count", [(16384, 64), (70_001, 33), (1 << 20, 12), (1 << 20, 31), (1 << 20, 32),
                                      (1 << 20, 97), (3_000_000, 33), (5_000_011, 31), (24_000_001, 65), (60_000_011, 40), (200_000_033, 24)])
def test_groups_equal_dense(eng, lo, count):
    ps = sieve.primes_from(lo, count)
    assert tup(eng.profiles(ps, mode="sparse", a4=False)) == tup(eng.profiles(ps, mode="dense", a4=False))


def test_groups_across_sizes_and_repeats(eng):
    """Primes of very different sizes, unsorted and with repeats, in one call."""
    ps = [p for k in range(14, 27) for p in sieve.primes_from((1 << k) + 12345, 9)]
    ps = ps[::-1] + ps[:20]
    assert tup(eng.profiles(ps, mode="sparse", a4=False)) == tup(eng.profiles(ps, mode="dense", a4=False))


def test_composite_among_grouped_primes_is_refused(eng):
    from rabung_atlas32_b200.census import CensusError
    t0 = time.perf_counter()
    with pytest.raises(CensusError, match="status"):
        eng.profiles(sieve.primes_from(1 << 25, 80) + [(1 << 25) + 1], mode="sparse", a4=True)
    assert time.perf_counter() - t0 < 5.0


@pytest.mark.parametrize("lo,count", [(3, 60), (16 * 1024 - 300, 40), (65_536 - 120, 30), (1 << 17, 20), (9_999_991, 3)])
def test_dense_scan_equals_oracle(eng, lo, count):
    """The dense scan on both sides of the least prime whose labels are kept,
    around one segment (8192 x) and one chunk, against the CPU oracle's walk."""
    import oracle
    ps = sieve.primes_from(lo, count)
    for r in eng.profiles(ps, mode="dense", a4=False):
        assert [(v.r, v.M, v.L, v.witness, v.K) for v in r.profiles] == \
               [(v["r"], v["max"], v["prefix"], v["witness"], v["K"]) for v in oracle.profiles(r.p)], r.p


@pytest.mark.parametrize("lo,count", [(2, 400), (990, 12), (16_777_259, 33), (4_294_960_000, 40)])
def test_a4_equals_oracle(eng, lo, count):
    """Point counts on both sides of the direct count's limit (p = 1000), and
    at odd batch sizes, against the CPU oracle."""
    import oracle
    ps = sieve.primes_from(lo, count)
    assert eng.a4(ps) == [oracle.a4(p) if p > 2 else 0 for p in ps]
