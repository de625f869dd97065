"""The autotuner against the launch plan: a form is chosen only where it is faster, and a kept
plan is saved and applied again (no GPU: the library and the timings are fakes)."""
import pytest

from gaussium_gb300 import autotune, engine


@pytest.fixture
def fake(monkeypatch):
    """(state of the chosen forms, run_class, times by (class, form, heavy form on))."""
    state, times, now = {}, {}, {}
    monkeypatch.setattr(autotune, "forms", lambda cls, prec: [1, 2] if cls[0] else [1])
    monkeypatch.setattr(autotune, "set_form", lambda cls, prec, v: state.__setitem__((cls, prec), v))
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: (fn(), now["t"])[1])

    def run_class(cls, prec):
        now["t"] = times[cls, state[cls, prec], (cls, prec) not in engine.SPLIT_OFF]

    def whole(prec):
        now["t"] = times["whole", tuple(state[c, prec] for c in (A, B, C))]
    run_class.whole = whole
    return state, run_class, times


A, B, C = (1, 0, 0, 0), (0, 0, 0, 0), (1, 1, 0, 0)


def test_plan_kept_unless_a_form_is_faster(fake, tmp_path):
    state, run_class, times = fake
    for cls, plan, t1, t2 in ((A, 1.0, 3.0, 0.99), (B, 1.0, 1.5, None), (C, 1.0, 2.0, 0.5)):
        times.update({(cls, 0, True): plan, (cls, 1, True): t1, (cls, 2, True): t2,
                      (cls, 1, False): t1 + 1, (cls, 2, False): (t2 or 0) + 1})
    engine.SPLIT_OFF.add((A, 64))                     # of an earlier choice
    segs = [(A, 0, 10), (B, 10, 20), (C, 20, 30)]
    tune = lambda: autotune.tune(segs, run_class, precisions=(64,), reps=1,     # noqa: E731
                                 whole=run_class.whole)
    times["whole", (0, 0, 0)], times["whole", (0, 0, 2)], times["whole", (2, 0, 2)] = 3.0, 2.5, 2.0
    chosen = tune()
    assert state == {(A, 64): 0, (B, 64): 0, (C, 64): 2} and not engine.SPLIT_OFF
    assert [chosen[c, 64]["plan"] for c in (A, B, C)] == [True, True, False]
    assert [autotune.describe(chosen[c, 64]) for c in (A, B, C)] == ["plan", "plan",
                                                                     "warp+cooperative"]
    assert chosen[A, 64]["form"] == 2 and set(chosen[A, 64]["ms"]) == {1, 2}
    # heavy quartets better left on the form: that time counts
    times[A, 2, False] = 0.5
    chosen = tune()
    assert state[A, 64] == 2 and not chosen[A, 64]["plan"] and engine.SPLIT_OFF == {(A, 64)}
    path = str(tmp_path / "forms.json")
    autotune.save(chosen, path)
    state.clear()
    engine.SPLIT_OFF.clear()
    again = autotune.load(path)
    assert state == {(A, 64): 2, (B, 64): 0, (C, 64): 2} and engine.SPLIT_OFF == {(A, 64)}
    assert again[B, 64]["plan"] and not again[C, 64]["plan"]
    # forms that are faster alone but hardly make the whole call faster: the plan for every class
    times["whole", (2, 0, 2)] = 2.95
    chosen = tune()
    assert all(r["plan"] for r in chosen.values()) and not engine.SPLIT_OFF
    assert state == {(A, 64): 0, (B, 64): 0, (C, 64): 0}


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
