"""The autotuner against the launch plan: a form is chosen only where it is faster, and a kept
plan is saved and applied again (no GPU: the library and the timings are fakes)."""
import pytest

from gaussium_gb300 import autotune, engine


@pytest.fixture
def fake(monkeypatch):
    """(state of the chosen forms, run_class, times by (class, form, heavy form on))."""
    state, times, now = {}, {}, {}
    monkeypatch.setattr(autotune, "forms", lambda cls, prec: [1, 2] if cls[0] else [1])
    monkeypatch.setattr(autotune, "set_form", lambda cls, prec, v: (
        state.__setitem__((cls, prec), v), engine.PLAN_ON.pop((cls, prec), None)))
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: (fn(), now["t"])[1])

    monkeypatch.setattr(engine, "PLAN_ON", {})
    planned = lambda k: engine.PLAN_ON.get(k) == state[k]        # noqa: E731

    def run_class(cls, prec):
        k = cls, prec
        now["t"] = times[cls, 0, True] if planned(k) else times[cls, state[k], k not in engine.SPLIT_OFF]

    def whole(prec):
        now["t"] = times["whole", tuple(0 if planned((c, prec)) else state[c, prec] for c in (A, B, C))]
    run_class.whole = whole
    return state, run_class, times


A, B, C = (1, 0, 0, 0), (0, 0, 0, 0), (1, 1, 0, 0)


def test_plan_kept_unless_a_form_is_faster(fake, tmp_path):
    state, run_class, times = fake
    for cls, plan, t1, t2 in ((A, 1.0, 3.0, 1.01), (B, 1.0, None, None), (C, 1.0, 2.0, 0.5)):
        times.update({(cls, 0, True): plan, (cls, 1, True): t1, (cls, 2, True): t2,
                      (cls, 0, False): plan + 1, (cls, 1, False): (t1 or 0) + 1,
                      (cls, 2, False): (t2 or 0) + 1})
    engine.SPLIT_OFF.add((A, 64))                     # of an earlier choice
    segs = [(A, 0, 10), (B, 10, 20), (C, 20, 30)]
    tune = lambda: autotune.tune(segs, run_class, precisions=(64,), reps=1,     # noqa: E731
                                 whole=run_class.whole)
    times["whole", (0, 0, 0)], times["whole", (0, 0, 2)], times["whole", (2, 0, 2)] = 3.0, 2.5, 2.0
    chosen = tune()
    # the forms are chosen (mixed builds take them), A's and B's plain calls follow the plan
    assert state == {(A, 64): 2, (B, 64): 0, (C, 64): 2} and not engine.SPLIT_OFF
    assert engine.PLAN_ON == {(A, 64): 2, (B, 64): 0}
    assert [chosen[c, 64]["plan"] for c in (A, B, C)] == [True, True, False]
    assert [autotune.describe(chosen[c, 64]) for c in (A, B, C)] == ["plan", "plan",
                                                                     "warp+cooperative"]
    assert chosen[A, 64]["form"] == 2 and set(chosen[A, 64]["ms"]) == {1, 2}
    # heavy quartets better left on the form: that time counts
    times[A, 2, False] = 0.5
    chosen = tune()
    assert state[A, 64] == 2 and not chosen[A, 64]["plan"] and engine.SPLIT_OFF == {(A, 64)}
    assert engine.PLAN_ON == {(B, 64): 0}
    path = str(tmp_path / "forms.json")
    autotune.save(chosen, path)
    for x in (state, engine.SPLIT_OFF, engine.PLAN_ON):
        x.clear()
    again = autotune.load(path)
    assert state == {(A, 64): 2, (B, 64): 1, (C, 64): 2} and engine.SPLIT_OFF == {(A, 64)}
    assert again[B, 64]["plan"] and not again[C, 64]["plan"] and engine.PLAN_ON == {(B, 64): 1}
    # forms that are faster alone but hardly make the whole call faster: the plan for every class
    times["whole", (2, 0, 2)] = 2.95
    chosen = tune()
    assert all(r["plan"] for r in chosen.values()) and engine.SPLIT_OFF == {(A, 64)}
    assert state == {(A, 64): 2, (B, 64): 0, (C, 64): 2} == engine.PLAN_ON


def test_launch_plan_of_a_class_left_to_the_plan(monkeypatch):
    """Plain calls of a class in PLAN_ON are cut into tiers while that form stays the chosen one; a
    form chosen afterwards counts; mixed builds follow the form."""
    import types
    import numpy as np
    import torch
    forms = {}

    class Library:
        def gs_class_variant(self, *a):
            return forms.get(a[4], 0)

        def gs_class_variants(self, *a):
            return 0b1111111

        def gs_class_form(self, *a):
            return forms.get(a[4], 0) or engine.WARP_FORM

        def gs_set_class_variant(self, *a):
            forms[a[4]] = a[5]
            return 0
    monkeypatch.setattr(engine._lib, "lib", Library)
    for name, value in (("SPLIT_OFF", set()), ("PLAN_ON", {})):
        monkeypatch.setattr(engine, name, value)
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d: types.SimpleNamespace(multi_processor_count=152))
    w = np.sort(np.random.default_rng(0).integers(1, 400, 5000))[::-1]
    e = types.SimpleNamespace(tasks=torch.zeros(1), segments=[(A, 0, 5000)], heavy=[engine.heavy_counts(A, w)],
                              profiles=[engine.work_profile(w)])
    plain = lambda: engine.launch_plan(e, 64, "jk")       # noqa: E731
    tiers = plain()
    autotune.set_form(A, 64, engine.STACKED_FORM)
    formed = plain()
    assert tiers != formed
    engine.PLAN_ON[A, 64] = engine.STACKED_FORM
    assert plain() == tiers and engine.mixed_plan(e, None, 1e-3)[0]
    autotune.set_form(A, 64, engine.STACKED_FORM)
    assert plain() == formed


def test_wrappers_compare_with_the_plan(monkeypatch):
    from gaussium_gb300.batch import BatchedRHF
    import torch
    seen = []
    monkeypatch.setattr(autotune, "tune", lambda *a, **kw: seen.append(callable(kw["whole"])))
    e = type("E", (), {"segments": [], "dev": torch.device("cpu")})()
    autotune.tune_jk(e, torch.zeros(1))
    autotune.tune_blocks(e, None)
    b = object.__new__(BatchedRHF)
    b.segments, b.mat_stride, b.dev = [], 1, torch.device("cpu")
    b.tune()
    assert seen == [True, True, True]
