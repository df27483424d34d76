"""Device memory: what a call allocates stays inside its plane budget, and a call
that can do with less runs where memory is short."""
import dataclasses

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def rows(c, ps, mode):
    out, _, _ = c.raw(ps, mode=mode, a4=False)
    return [(o.p, o.r, o.M, o.L, o.witness, o.K) for o in out]


@pytest.fixture(scope="module")
def tuned():
    from rabung_atlas32_b200.census import Census
    with Census() as c:
        yield c.tuning


def test_dense_labels_inside_the_plane_budget(tuned):
    """100 primes near 2^24 keep 0.77 GB of labels where the budget allows."""
    from rabung_atlas32_b200.census import Census
    ps = sieve.primes_from(1 << 24, 100)
    with Census() as c:
        want = rows(c, ps, "dense")
    with Census(tuning=dataclasses.replace(tuned, plane_budget_mb=64)) as c:
        rows(c, ps[:1], "dense")                          # static tables and small buffers are there
        before = c.mem_info()[0]
        assert rows(c, ps, "dense") == want
        assert before - c.mem_info()[0] < (64 + 32) << 20
    with Census(tuning=dataclasses.replace(tuned, plane_budget_mb=4)) as c:
        assert rows(c, ps[:20], "dense") == want[:len(rows(c, ps[:20], "dense"))]      # no prime's labels fit


def test_dense_scan_where_labels_do_not_fit_the_device(tuned):
    """All but 0.5 GB of the device is taken; the labels of 300 primes near 2^24
    would take 2 GiB."""
    import torch
    from rabung_atlas32_b200.census import Census
    ps = sieve.primes_from(1 << 24, 300)
    with Census() as c:
        want = rows(c, ps, "auto")
    with Census(tuning=tuned) as c:
        rows(c, ps[:1], "dense")
        torch.cuda.empty_cache()
        free = c.mem_info()[0]
        hold = torch.empty(free - (512 << 20), dtype=torch.uint8, device="cuda")
        try:
            assert rows(c, ps, "dense") == want
            assert rows(c, ps[:5], "auto") == want[:len(rows(c, ps[:5], "auto"))]      # the next call is not affected
        finally:
            del hold
            torch.cuda.empty_cache()


def test_scattered_groups_inside_the_plane_budget(tuned):
    """Ten windows of 10 primes, a factor of 2 apart: groups of 4 to 10 members,
    which take up to four times their members' own planes."""
    from rabung_atlas32_b200.census import Census
    ps = [p for k in range(10) for p in sieve.primes_from(4200000000 >> k, 10)]
    with Census(tuning=tuned) as c:
        need = c.plane_bytes(ps, mode="sparse") >> 20
        want = rows(c, ps, "sparse")
        assert c.last_stats["kernels"] > 10               # groups were formed
    with Census(tuning=dataclasses.replace(tuned, plane_budget_mb=need + 1)) as c:
        rows(c, ps[:1], "sparse")
        before = c.mem_info()[0]
        assert rows(c, ps, "sparse") == want
        assert c.last_stats["waves"] == 1
        # planes, the labels beside them (a sixteenth) and the buffers' slack of a quarter
        assert before - c.mem_info()[0] < need * 1.4 * 2 ** 20


def test_server_whose_arena_takes_the_device(tuned):
    """An arena capped by the free memory leaves 4 GiB beside it.  In these: two
    requests of 34,000 primes near 2^24, which run in one joint call, and one of
    4096 primes near 2^32, which stays resident."""
    from rabung_atlas32_b200.census import Census
    from rabung_atlas32_b200.serving import Server
    reqs = [(1 << 24, 34000), (15_000_000, 34000), (4_200_000_000, 4096)]
    srv = Server(slots=16, slot_budget_mb=24 * 1024, tuning=tuned)
    try:
        ids = [srv.submit(lo, n) for lo, n in reqs]
        got = [srv.fetch(rid, n) for rid, (lo, n) in zip(ids, reqs)]
    finally:
        srv.close()
    with Census(tuning=tuned) as c:
        for (lo, n), (primes, recs) in zip(reqs, got):
            assert primes == sieve.primes_from(lo, n)
            assert [(r.p, v.r, v.M, v.L, v.witness, v.K) for r in recs for v in r.profiles] == rows(c, primes, "auto")


def test_planes_and_labels_share_the_budget(tuned):
    """One call with 100 sparse primes near 2^28 and 100 dense ones near 2^24
    (sparse_min_p between them): 0.05 GB of planes, 0.77 GB of labels."""
    from rabung_atlas32_b200.census import Census
    ps = sieve.primes_from(1 << 24, 100) + sieve.primes_from(1 << 28, 100)
    t = dataclasses.replace(tuned, sparse_min_p=1 << 26)
    with Census(tuning=t) as c:
        want = rows(c, ps, "auto")
        assert c.last_stats["n_dense"] == 100 and c.last_stats["n_sparse"] == 100
        planes = c.plane_bytes(ps, mode="auto") >> 20
    with Census(tuning=dataclasses.replace(t, plane_budget_mb=planes + 32)) as c:
        rows(c, ps[:1], "dense")
        before = c.mem_info()[0]
        assert rows(c, ps, "auto") == want
        assert before - c.mem_info()[0] < (planes + 32) * 1.4 * 2 ** 20 + (8 << 20)
