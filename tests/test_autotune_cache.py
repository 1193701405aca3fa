"""The tuner's cache (no GPU: a model and a batch that take any schedule, and a
clock that likes one of them): choices cached when the schedules' names meant
other kernels are not taken; its own are."""
import json

import pytest

from raytracer_3d_gb300 import autotune

N = (8, 8, 8, 6, 6, 8)


class _Lib:
    def rt_step_dry(self, h, k):
        return 0

    def rt_batch_dry(self, b, k):
        return 0


class _Model:
    n, precision, handle, _b = N, "fp32", None, None

    def __init__(self):
        self._lib, self.now = _Lib(), None
        self.models = [self]

    def stream(self):
        return 0

    def _check(self, rc, what):
        pass

    def set_tuning(self, *c):
        self.now = tuple(c)

    def set_persistent(self, t):
        self.now = self.now[:3] + (t,)

    def set_slices(self, t):
        pass

    def set_fused(self, on):
        pass


@pytest.fixture
def cache(tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("RT_TUNE_CACHE", str(path))
    monkeypatch.setattr(autotune, "_event_timer", lambda stream: lambda fn, reps: fn(reps) or 1.0)
    return path


def test_older_model_choice_is_not_taken(cache):
    name = "x".join(map(str, N))
    cache.write_text(json.dumps({"model|fp32|" + name: {"best": ["w3", 8, 256, 0], "table": []}}))
    m = _Model()
    best, _ = autotune.tune_model(m, candidates=[("tma", 8, 512, 0)])
    assert best == ("tma", 8, 512, 0) and m.now == best
    other = _Model()
    assert autotune.tune_model(other, candidates=[("w2z", 8, 512, 0)])[0] == best and other.now == best   # its own


def test_older_batch_choice_is_not_taken(cache):
    name = "x".join(map(str, N))
    cache.write_text(json.dumps({"batch4|fp32|" + name: {"best": [8, 512, 1, 512, 512, 1], "table": []}}))
    b = _Model()
    best, _ = autotune.tune_batch(b, candidates=[(4, 512, 0, 0, 0, 0)])
    assert best == (4, 512, 0, 0, 0, 0) and b.now == (4, 512, 0, 0)
    assert autotune.tune_batch(_Model(), candidates=[(8, 512, 0, 256, 256, 0)])[0] == best
