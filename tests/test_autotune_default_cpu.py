"""The autotuner's candidates hold the engine's own choice, so that a tuned
handle is never slower than a plain one by more than the timing's noise; cached
entries from a list without it are timed again."""
import json

import pytest

import titan_gb300 as tg
from titan_gb300 import autotune as at
from titan_gb300 import workloads as wl


@pytest.mark.parametrize("prec", [tg.FP64, tg.FP32, tg.FP32C])
def test_the_default_is_a_candidate(monkeypatch, tmp_path, prec):
    calls = []

    def fake_time(sc, precision, cand, steps, device):
        calls.append(tuple(cand))
        return (0.1 if tuple(cand) == (0, 0, 0) else 0.2), "per-tile"

    monkeypatch.setattr(at, "_time_candidate", fake_time)
    monkeypatch.setattr(at, "_gpu_name", lambda device: "test-gpu")
    sc = wl.actuated_lattice(n_side=6)
    cache = tmp_path / "tune.json"
    old = {"kernel": 1, "tile": 128, "threads": 128, "ms_per_step": 0.2, "form": "per-tile",
           "tried": [{"candidate": [1, 128, 128], "ms_per_step": 0.2, "form": "per-tile"}]}
    cache.write_text(json.dumps({at.scene_key(sc, prec): old}))
    best = at.autotune(sc, prec, cache_path=cache)
    assert (best["kernel"], best["tile"], best["threads"]) == (0, 0, 0) and calls.count((0, 0, 0)) == 1
    n = len(calls)
    assert at.autotune(sc, prec, cache_path=cache)["kernel"] == 0 and len(calls) == n  # from the cache
    assert at.autotune(sc, prec, candidates=[(1, 128, 128)], cache_path=cache)["kernel"] == 0 and len(calls) == n
