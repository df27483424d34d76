"""Counters of a call: the bytes copied back are those of the one copy that is made
(records, A4, per-profile state), and those of its re-runs."""
import dataclasses

import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


def test_bytes_copied_back():
    from rabung_atlas32_b200.census import Census
    ps = sieve.primes_ending(1 << 28, 64)
    with Census() as c:
        tuned = c.tuning
    stats = []
    for shift in (20, None):                                  # wide margins: no re-runs; none: many
        margins = tuple(m + shift if shift else 0 for m in tuned.spec_margin10)
        with Census(tuning=dataclasses.replace(tuned, spec_margin10=margins)) as c:
            stats.append(c.raw(ps, mode="sparse", a4=True)[2])
    plain, rerun = stats
    assert plain["n_respec"] == 0 and rerun["n_respec"] > 0
    # a record (32 bytes) and a state (64) per profile, an A4 count (4) per prime
    least = 96 * plain["n_profiles"] + 4 * len(ps)
    assert least <= plain["d2h_bytes"] < least + 2048
    assert rerun["d2h_bytes"] > plain["d2h_bytes"] and rerun["h2d_bytes"] > plain["h2d_bytes"]
