"""The batch autotuner: candidates that differ, timings of another kernel not reused (no GPU)."""
import json

import numpy as np

from taichi_lbm3d_gb300 import autotune


class FakeBatch:
    def __init__(self, solids, **kw):
        self.n = len(solids)

    def info(self):
        return {"n_fluid": 1000}

    def close(self):
        pass


def tune(monkeypatch, path, ms, **kw):
    from taichi_lbm3d_gb300 import batch
    timed = []

    def time_config(b, tile, block, **kw):
        timed.append((tile, block))
        return ms(tile, block)

    monkeypatch.setattr(batch, "Batch", FakeBatch)
    monkeypatch.setattr(autotune, "time_config", time_config)
    monkeypatch.setattr(autotune, "_gpu_name", lambda: "gpu")
    s = np.zeros((4, 4, 4), np.int8)
    return autotune.tune({48: [s], 160: [s]}, storage="f16", path=path, **kw), timed


def test_candidates_are_different_launches(monkeypatch, tmp_path):
    """The kernel takes tiles in whole groups of 32 nodes, at most the CTA's threads."""
    _, timed = tune(monkeypatch, str(tmp_path / "t.json"), lambda t, b: 1.0)
    made = [(min((max(32, t) + 31) // 32 * 32, b), b) for t, b in timed]
    assert len(set(made)) * 2 == len(made)          # two edge classes, every launch once
    assert len({t for t, _ in made}) >= 3 and len({b for _, b in made}) >= 3


def test_timings_of_another_kernel_are_not_served(monkeypatch, tmp_path):
    path = str(tmp_path / "t.json")
    old = {"tile": 1024, "block": 256, "ms_per_step": 0.1, "when": "before"}
    with open(path, "w") as fh:
        json.dump({"gpu|f16|48": old, "gpu|f16|160": old}, fh)
    res, timed = tune(monkeypatch, path, lambda t, b: 1.0 + 0.1 * (b != 128) + 0.01 * (t != b))
    assert timed and (res[48]["tile"], res[48]["block"]) == (128, 128)
    again, timed = tune(monkeypatch, path, lambda t, b: 0.0)
    assert not timed and again == res


def test_plan_takes_the_fastest_tile_of_its_block():
    tuned = {48: {"tile": 64, "block": 64, "trials_ms": {"64/64": 1.0, "64/128": 1.3, "128/128": 1.2, "128/64": 9.0}},
             160: {"tile": 128, "block": 128, "trials_ms": {"64/64": 2.0, "64/128": 2.1, "128/128": 1.9}}}
    assert autotune.plan([48, 160, 48], tuned) == ([128, 128, 128], 128)
    assert autotune.plan([48, 48], tuned) == ([64, 64], 64)
