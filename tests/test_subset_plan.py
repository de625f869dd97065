"""Launch plans of calls for some of an engine's classes."""
import types

import numpy as np
import torch

from gaussium_gb300 import engine


def test_tiers_of_a_small_class_alone(monkeypatch):
    """Alone, no tier's longest task of a small class takes longer than twice the class's work (or
    the shortest time worth splitting), whatever the other classes would take; with them it may."""
    class Stub:
        def gs_class_variant(self, *a):
            return 0

        def gs_class_variants(self, *a):
            return 0b1111111
    monkeypatch.setattr(engine._lib, "lib", Stub)
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d: types.SimpleNamespace(multi_processor_count=152))
    rng = np.random.default_rng(0)
    small, large = (1, 0, 0, 0), (2, 2, 2, 2)
    e = types.SimpleNamespace(tasks=torch.zeros(1), segments=[], profiles=[], heavy=[])
    for cls, n, at in ((small, 10000, 0), (large, 400000, 10000)):
        w = np.sort(rng.integers(1, 300, n))[::-1]
        e.segments.append((cls, at, at + n))
        e.profiles.append(engine.work_profile(w))
        e.heavy.append(engine.heavy_counts(cls, w))
    longest = lambda *a: max(lat for c, *_, lat in engine.launch_plan(e, *a) if c == small)  # noqa: E731
    alone = engine.total_slots(e.segments[:1], e.profiles[:1], 64, "write", 608)
    bound = max(engine.MIN_LATENCY, engine.ALONE_SHARE * alone)
    assert longest(64, "write") > bound >= longest(64, "write", [small])
    plan = engine.launch_plan(e, 64, "write", [small])
    assert sum(n for _, _, n, _, _ in plan) == 10000
    assert engine.launch_plan(e, 64, "write", [(0, 0, 0, 0)]) == []
    # what mixed plans ask for, a class within the whole build, is not cut
    whole = [x for x in engine.launch_plan(e, 64, "jk", None, 0.5) if x[0] == small]
    assert sorted(engine.launch_plan(e, 64, "jk", [small], 0.5)) == sorted(whole)
