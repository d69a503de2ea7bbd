"""The autotuner's choice and its cache (CPU, no kernels): entries timed under another launch table are
not taken, and the default is not given up to noise."""
import json
import types

import torch

from altar_gb300 import _native, autotune


class _Lib:
    def ag_forward_variants(self, kind):
        return 3


class _Strategy:
    """Three launch variants that take the given times on a fake clock."""

    def __init__(self, clock, times):
        self.kind = _native.AG_MODEL_CDM
        self.stations = types.SimpleNamespace(m=40)
        self.layout = types.SimpleNamespace(variant=0)
        self.clock, self.times, self.calls = clock, times, 0

    def forward(self, theta, out):
        self.calls += 1
        self.clock[0] += self.times[self.layout.variant]


def _fake_gpu(monkeypatch, clock):
    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self, stream=None):
            self.at = clock[0]

        def elapsed_time(self, other):
            return other.at - self.at

    monkeypatch.setattr(_native, "load", lambda: _Lib())
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: None)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda: "GPU")


def test_entry_of_another_launch_table_is_ignored(monkeypatch, tmp_path):
    path = tmp_path / "autotune.json"
    monkeypatch.setenv("ALTAR_GB300_TUNE_CACHE", str(path))
    clock = [0.0]
    _fake_gpu(monkeypatch, clock)
    theta = torch.zeros(10, 4, dtype=torch.float64)
    # as the cache was written before the table had a number
    path.write_text(json.dumps({"model=2 m=40 n=10 variants=3 gpu=GPU": {"variant": 1, "ms": [3.0, 1.0, 2.0]}}))
    strategy = _Strategy(clock, [1.0, 3.0, 2.0])
    assert autotune.tune(strategy, theta)["variant"] == 0 and strategy.layout.variant == 0 and strategy.calls > 0
    # this table's own entry is taken without a trial
    again = _Strategy(clock, [9.0, 9.0, 1.0])
    assert autotune.tune(again, theta)["variant"] == 0 and again.calls == 0
    # and no longer once the table changes
    monkeypatch.setattr(autotune, "LAUNCH_TABLE", autotune.LAUNCH_TABLE + 1)
    assert autotune.tune(again, theta)["variant"] == 2 and again.calls > 0


def test_default_is_kept_against_noise(monkeypatch, tmp_path):
    """Two variants that are one kernel (14.374 and 14.368 ms, measured): the choice is not their noise."""
    monkeypatch.setenv("ALTAR_GB300_TUNE_CACHE", str(tmp_path / "autotune.json"))
    clock = [0.0]
    _fake_gpu(monkeypatch, clock)
    theta = torch.zeros(10, 4, dtype=torch.float64)
    for times, want in (([14.374, 15.0, 14.368], 0), ([14.368, 15.0, 14.374], 0), ([14.4, 14.0, 14.2], 1)):
        strategy = _Strategy(clock, times)
        assert autotune.tune(strategy, theta, use_cache=False)["variant"] == want
        assert strategy.layout.variant == want
