"""The batch autotuner's cache: a choice made for an older kernel is not applied."""
import json

import torch

from verona_b200 import autotune


class _Batch:
    precision = 1
    tuning = {"grid": 1}

    def __init__(self):
        self.applied = []

    def set_tuning(self, variant, ctas):
        self.applied.append((variant, ctas))

    def signature(self):
        return "abc"

    def _nothing(self, *a):
        pass

    checkpoint = rollback = step = reset_counters = _nothing


class _Event:
    def __init__(self, **k):
        pass

    def record(self, stream):
        pass

    def elapsed_time(self, other):
        return 1.0


def _tune(monkeypatch, path):
    monkeypatch.setattr(autotune, "_gpu_key", lambda: "gpu/sm100/148")
    monkeypatch.setattr(autotune, "variants", lambda precision: ["a", "b"])
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: None)
    monkeypatch.setattr(torch.cuda, "Event", _Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    b = _Batch()
    return b, autotune.tune_batch(b, path=str(path))


def test_choice_of_an_older_kernel_is_made_again(monkeypatch, tmp_path):
    path = tmp_path / "tune.json"
    old = {"variant": 1, "ctas_per_sm": 2, "shape": "b", "ms_per_step": 0.1}
    path.write_text(json.dumps({"gpu/sm100/148/abc": old, "gpu/sm100/148/k1/abc": old}))
    b, r = _tune(monkeypatch, path)
    assert not r["cached"] and len(b.applied) > 2  # every candidate was tried
    b, r = _tune(monkeypatch, path)
    assert r["cached"] and len(b.applied) == 1  # and the new choice is kept
    assert json.loads(path.read_text())["gpu/sm100/148/abc"] == old  # other entries stay
