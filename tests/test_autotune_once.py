"""The autotuner times a program once: candidates that differ only in the option without effect
share one measurement, so that noise cannot choose between them."""

from __future__ import annotations

import itertools

from galaxy_collision_gb300 import autotune


def test_equal_programs_are_timed_once(tmp_path, monkeypatch):
    noise = itertools.count()
    seen = []

    def fake(make_engine, state, dt, settings, steps=20, warm=3):
        seen.append(settings["sort_every"])
        return {20: 3.0, 10: 2.0}[settings["sort_every"]] - 1e-3 * next(noise)  # every timing a little lower

    monkeypatch.setattr(autotune, "time_candidate", fake)
    e = autotune.tune(64, 300_000, None, None, 0.005, device="dev", path=tmp_path / "tune.json")
    assert sorted(seen) == sorted({c["sort_every"] for c in autotune.CANDIDATES})
    assert len(e["ms_per_step"]) == len(autotune.CANDIDATES)
    assert e["settings"] == {"phase_launches": False, "sort_every": 10}
