"""Tuning fields that act also in calls whose profiles would be filtered in groups:
the screen (without it there are no groups) and the number of CTAs.  The records
stay."""
import dataclasses

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def run(tuning, ps):
    from rabung_atlas32_b200.census import Census
    with Census(tuning=tuning) as c:
        for _ in range(2):
            out, _, st = c.raw(ps, mode="sparse", a4=False)
        return [(o.p, o.r, o.M, o.L, o.witness, o.K) for o in out], st


def test_screen_and_sparse_blocks_act():
    """64 times one prime: two full groups of every order, nothing beside them."""
    from rabung_atlas32_b200.census import Census
    with Census() as c:
        tuned = c.tuning
    ps = sieve.primes_from(1 << 26, 1) * 64
    want, st = run(tuned, ps)
    got, bare = run(dataclasses.replace(tuned, screen=0), ps)
    assert got == want and bare["completions"] > 2 * st["completions"]
    got, one = run(dataclasses.replace(tuned, sparse_blocks=1), ps)
    assert got == want and one["ms_sparse"] > 10 * st["ms_sparse"]
