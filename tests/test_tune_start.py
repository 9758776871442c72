"""The tuner starts from the untuned plan, so its choice is never one that it
measured slower than that plan, and its default_ms is that plan's (host logic only:
the timing is replaced)."""
import json

import pytest
import torch

from crossstage_stitch_b200 import tune


@pytest.fixture
def tuner(tmp_path, monkeypatch):
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "a GPU")
    return tune.Tuner(tmp_path / "tuning.json", device="cuda:0")


def test_untuned_plan_is_kept_when_nothing_is_faster(tuner, monkeypatch):
    timed = []

    def time_plan(pairs, tuning):
        timed.append(dict(tuning))
        return 1.0 if not any(tuning.values()) else 1.5
    monkeypatch.setattr(tuner, "time_plan", time_plan)
    assert not any(tuner.tune(("vga", "k500"), [None]).values())
    assert not any(timed[0].values()) and all(any(t.values()) for t in timed[1:])
    entry = json.loads(tuner.path.read_text())["a GPU|vga|k500"]
    assert entry["default_ms"] == entry["tuned_ms"] == 1.0


def test_faster_shapes_are_found_from_the_untuned_plan(tuner, monkeypatch):
    gain = {("resize_tile_h", 64): 0.1, ("resize_tile_h", 32): 0.2, ("blur_ctas_per_sm", 6): 0.1, ("search_hpw", 32): 0.3}
    monkeypatch.setattr(tuner, "time_plan", lambda pairs, t: 2.0 - sum(gain.get(kv, -0.05 if kv[1] else 0.0) for kv in t.items()))
    got = tuner.tune(("4k", "k8000"), [None])
    assert got == {"fast_ctas_per_sm": 0, "resize_tile_h": 32, "blur_ctas_per_sm": 6, "matcher": 0, "search_hpw": 32}
    assert tuner.table["a GPU|4k|k8000"]["default_ms"] == 2.0
