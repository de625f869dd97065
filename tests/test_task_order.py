"""Task order of contractions whose pairs keep 64 primitive pairs and more."""
import numpy as np
import pytest
import torch


def test_batched_order_of_long_contractions():
    """Work never rises along a segment: the launch plans' profiles search it."""
    from gaussium_gb300.batch import batched_task_list
    rng = np.random.default_rng(2)
    n = 120
    nprim = torch.as_tensor(rng.choice([1, 2, 63, 64, 65, 90, 4096, 8000], n))
    q, zero = torch.ones(n, dtype=torch.float64), torch.zeros(n, dtype=torch.int64)
    segs, tasks = batched_task_list(q, zero, zero, nprim, 0.0, 1, 1)
    assert len(segs) == 1 and len(tasks) == n * (n + 1) // 2
    work = (nprim[tasks[:, 0].long()] * nprim[tasks[:, 1].long()]).numpy()
    assert np.all(np.diff(work) <= 0)


@pytest.mark.gpu
def test_task_keys_of_long_contractions(gpu_lib):
    """The key's upper part is the primitive-quartet count and the order follows it."""
    from gaussium_gb300 import engine
    from gaussium_gb300.basis import ShellBasis
    rng = np.random.default_rng(5)
    shells = [dict(l=0, centre=rng.uniform(-1, 1, 3), expo=np.exp(rng.uniform(-2, 3, k)),
                   coef=rng.uniform(0.2, 1.0, k)) for k in (1, 2, 7, 8, 9, 13)]
    eng = engine.JKEngine(ShellBasis.from_shell_dicts(shells), schwarz_thr=0.0, max_exp=0.0)
    nprim = eng.pairs.nprim
    assert nprim.max() == 169
    t = eng.tasks[:eng.ntasks].long()
    keys = engine.task_keys(eng.pairs, t[:, 0].contiguous(), t[:, 1].contiguous()).cpu().numpy()
    work = nprim[t[:, 0].cpu()] * nprim[t[:, 1].cpu()]
    assert np.array_equal(keys // engine.KEY_WORK, work) and np.array_equal(keys >> 18, work)
    assert np.all(np.diff(work) <= 0)
    assert eng.profiles[0] == engine.work_profile(work)


@pytest.mark.parametrize("at_once", [1 << 26, 10])
@pytest.mark.parametrize("first", [0, 7])
def test_segment_profiles_of_uneven_segments(monkeypatch, at_once, first):
    """Empty and one-task segments, counts of zero and far beyond the levels, a list that starts
    behind others, and lists taken segment by segment: the host's counts."""
    from gaussium_gb300 import engine
    monkeypatch.setattr(engine, "SEARCH_AT_ONCE", at_once)
    rng = np.random.default_rng(6)
    segs = [np.sort(rng.integers(0, t, n))[::-1] for t, n in
            ((1, 5), (1300, 400), (2, 0), (1 << 45, 30), (5, 1), (129, 200), (1, 0))]
    cls = [(0, 0, 0, 0), (2, 2, 2, 2), (1, 0, 0, 0), (1, 1, 1, 1), (2, 0, 0, 0), (2, 1, 1, 0), (1, 1, 0, 0)]
    w = torch.as_tensor(np.concatenate([np.full(first, 99), *segs]))
    bounds = (first + np.concatenate([[0], np.cumsum([len(x) for x in segs])])).tolist()
    got = engine.segment_profiles(cls, w, bounds)
    assert got == [(engine.heavy_counts(c, x), engine.work_profile(x)) for c, x in zip(cls, segs)]
    assert engine.segment_profiles([], w, [0]) == []
