"""A cached launch shape stands only for the kernels and the shapes it was timed against."""

from __future__ import annotations

from test_datagen_host import _FakeEngine


class _OneMoreShape(_FakeEngine):
    def shape_candidates(self, which):
        return [*super().shape_candidates(which), (3, 640, 8)]


def _tune(autotune, monkeypatch, eng, path, ms):
    monkeypatch.setattr(autotune, "device_tag", lambda: "GB300-test|sm152")
    monkeypatch.setattr(autotune, "_probe_models", lambda eng, models, seed: object())
    monkeypatch.setattr(autotune, "_time_forward", lambda eng, vel, reps: ms[eng.shape["forward"]])
    return autotune.tune(eng, which=("forward",), path=path)["forward"]


def test_a_shape_added_since_is_timed(tmp_path, monkeypatch):
    from wgnet_gb300 import autotune

    path = tmp_path / "tune.json"
    ms = {(2, 704, 10): 3.0, (2, 896, 8): 2.5, (4, 448, 8): 4.0, (3, 640, 8): 2.0}
    assert _tune(autotune, monkeypatch, _FakeEngine(), path, ms) == (2, 896, 8)
    assert _tune(autotune, monkeypatch, _OneMoreShape(), path, ms) == (3, 640, 8)
    assert _tune(autotune, monkeypatch, _FakeEngine(), path, {}) == (2, 896, 8)  # still cached


def test_other_kernels_are_timed_again(tmp_path, monkeypatch):
    from wgnet_gb300 import autotune

    path = tmp_path / "tune.json"
    ms = {(2, 704, 10): 3.0, (2, 896, 8): 2.5, (4, 448, 8): 4.0}
    assert _tune(autotune, monkeypatch, _FakeEngine(), path, ms) == (2, 896, 8)
    monkeypatch.setattr(autotune, "kernels_tag", lambda: "other")
    assert _tune(autotune, monkeypatch, _FakeEngine(), path, ms | {(2, 704, 10): 1.0}) == (2, 704, 10)
