"""The autotuner's choice of a stack depth, with made-up times."""
import pytest


class _Scene:
    def set_tuning(self, **cfg):
        self.cfg = cfg


@pytest.mark.parametrize("shallow_ms,depth", [(0.995, 96), (0.991, 96), (0.98, 48), (0.5, 48), (1.2, 96)])
def test_shallow_stacks_must_pay(built, monkeypatch, shallow_ms, depth):
    """48 entries are kept when they are more than 1% faster than the default
    96; level with it the default stays, and the time reported is its own."""
    import torch

    import treelet_rt as rt
    from treelet_rt import autotune as at

    def time_trace(scene, *_):
        return {48: shallow_ms, 96: 1.0, 160: 1.1}[scene.cfg["stack_depth"]] + (scene.cfg["refill_lanes"] != 16) * 0.1

    monkeypatch.setattr(at, "time_trace", time_trace)
    monkeypatch.setattr(at, "_overflowed", lambda *_: False)
    scene = _Scene()
    r = at.autotune(scene, torch.zeros(32, dtype=torch.uint8), 1, rt.MODE_TREELET)
    assert r["tuning"]["stack_depth"] == depth and r["tuning"]["refill_lanes"] == 16
    assert r["ms"] == pytest.approx(1.0 if depth == 96 else shallow_ms)
    assert scene.cfg["stack_depth"] == depth
