"""A replay after calls that were refused: the last good call's plan is still
resident, its groups included."""
import pytest

from rabung_atlas32_b200 import sieve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("bad,mode", [([1], "auto"), ([5, 7, 11], "sparse")])
def test_replay_after_a_refused_call(use_graph, bad, mode):
    """A prime out of the domain and one without a sparse route, before the
    first replay of a call whose profiles are filtered in groups."""
    import dataclasses
    from rabung_atlas32_b200.census import Census, CensusError
    with Census() as probe:
        margins = tuple(m + 20 for m in probe.tuning.spec_margin10)       # no re-runs in this call
        tuning = dataclasses.replace(probe.tuning, use_graph=use_graph, spec_margin10=margins)
    ps = sieve.primes_ending(1 << 28, 64)
    with Census(tuning=tuning) as c:
        _, _, st = c.raw(ps, mode="sparse", a4=False)
        assert st["n_respec"] == 0 and st["kernels"] > 10                 # grouped: tables by level
        with pytest.raises(CensusError):
            c.raw(bad, mode=mode, a4=False)
        again = c.replay()
        assert again["n_profiles"] == st["n_profiles"] and again["n_sparse"] == len(ps)
        assert again["kernels"] == st["kernels"]
