"""Saved launch shapes of the batched day."""
import json
import types


def test_shapes_timed_on_earlier_kernels_are_not_taken(tmp_path, monkeypatch):
    from solweig_cuda_b200 import _lib, tune
    monkeypatch.setenv("SOLWEIG_TUNE_CACHE", str(tmp_path / "tune.json"))
    monkeypatch.setattr(tune.torch.cuda, "get_device_name", lambda device=None: "device")
    runner = types.SimpleNamespace(hours=24, scene=types.SimpleNamespace(
        device=None, rows=500, cols=500, struct=types.SimpleNamespace(patches=153)))
    key = tune.tune_key(runner)
    shapes = list(_lib.SolweigDayConfig.default().astuple())
    old = "v5" + key[key.index("|"):]  # before the walk-word GVF and the packed sweep
    (tmp_path / "tune.json").write_text(json.dumps({old: {"config": shapes, "stage_ms": {}}}))
    assert tune.lookup(runner) is None
    (tmp_path / "tune.json").write_text(json.dumps({key: {"config": shapes, "stage_ms": {}}}))
    assert list(tune.lookup(runner).astuple()) == shapes
