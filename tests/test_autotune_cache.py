"""The autotuner's cache against variant numbers that changed their meaning (no device)."""

import types

import torch

from symcode import autotune as A


def test_a_choice_of_an_earlier_kernel_set_is_timed_again(tmp_path, monkeypatch):
    path = str(tmp_path / "tune.json")
    g = types.SimpleNamespace(D=3, n=128, dtype=torch.float32, device="cuda:0")
    counts, applied = [3, 3, 2, 3, 3], []
    timings = {0: {s: 1.0 for s in A.SWEEPS}, 1: {s: 2.0 for s in A.SWEEPS}}
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "NVIDIA B200")
    monkeypatch.setattr(A, "num_variants", lambda g: counts)
    monkeypatch.setattr(A, "set_variants", lambda g, v: applied.append(v))
    monkeypatch.setattr(A, "measure", lambda *a: timings)
    # as stored before the x sweeps of 64 and 128 were renumbered: 1 was the faster one
    A.save_cache(path, "NVIDIA B200|D=3|n=128|float32", {"variants": {s: 1 for s in A.SWEEPS}, "ms": {}})
    assert A.tune(g, cache=path)["source"] == "timed"
    assert applied[-1] == {s: 0 for s in A.SWEEPS}
    assert A.tune(g, cache=path)["source"] == "cache"
    monkeypatch.setattr(A, "KERNEL_SET", A.KERNEL_SET + 1)
    assert A.tune(g, cache=path)["source"] == "timed"
