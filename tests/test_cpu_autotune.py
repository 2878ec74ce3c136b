"""tune_batch times every kernel variant once (a fake batch and clock, no GPU)."""
import torch

from diffsplat_b200 import _lib as L, api, autotune


def test_each_variant_is_timed_once(monkeypatch):
    made = []

    class Batch:
        def __init__(self, sizes, **kw):
            made.append((kw["tile_size"], kw["schedule"]))

        def step(self, n):
            pass

        def status(self):
            return L.DS_OK, 0

        def close(self):
            pass

    class Event:
        def __init__(self, enable_timing):
            pass

        def record(self):
            pass

        def elapsed_time(self, other):
            return 6.0 if made[-1] == (8, L.DS_SCHEDULE_RASTER) else 12.0

    monkeypatch.setattr(api, "Batch", Batch)
    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda: None)
    best, table = autotune.tune_batch([(64, 64, 100)], lambda b: None)
    assert len(made) == len(set(made)) == len(table) == 6
    assert best == dict(tile_size=8, ppt=1, schedule=L.DS_SCHEDULE_RASTER)
