"""The autotuner measures a knob where it acts: the stages, epochs and CTAs of the
per-profile filter in calls without speculation (grouped profiles read none of
them), the cover and the margins with it."""
from rabung_atlas32_b200 import autotune
from rabung_atlas32_b200.census import Tuning

RECORDS = [(101, 2, 7, 1, 19)]


def test_per_profile_knobs_are_measured_without_speculation(monkeypatch):
    base = Tuning()

    def model(t: Tuning, primes, mode: str, reps: int = 2):
        if mode == "dense":
            return 100.0, RECORDS
        ms = 1000.0 + 20.0 * abs(t.cover_n - 4)
        if t.speculate:
            # grouped: a few percent of noise that favours some settings
            ms -= 30.0 * (t.epoch_rows == 256) + 30.0 * (t.cta_per_profile == 4) + 30.0 * (t.anchor_t[2] == 10)
        else:
            ms += 40.0 * (t.epoch_rows != 2048) + 40.0 * abs(t.cta_per_profile - 2) + 40.0 * abs(t.anchor_t[2] - 12)
        return ms, RECORDS

    monkeypatch.setattr(autotune, "_measure", model)
    t = autotune.tune(quick=True, log=lambda s: None)["tuning"]
    assert (t["epoch_rows"], t["cta_per_profile"], t["anchor_t"][2]) == (2048, 2, 12)
    assert t["cover_n"] == 4 and t["speculate"] == base.speculate
