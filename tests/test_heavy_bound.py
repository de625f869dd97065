"""Batched mixed builds: quartets of many primitive quartets take the molecule's largest |P| for
their bound, the others the largest of their six shell blocks."""
import types

import numpy as np
import pytest
import torch

from gaussium_gb300 import engine


def test_tiers_of_the_heavy_prefix_carry_the_bound(monkeypatch):
    c1, c2 = (2, 1, 1, 0), (1, 0, 0, 0)
    plans = {64: [(c1, 0, 5, 7, 9.0), (c1, 5, 95, 6, 1.0)], 32: [(c1, 0, 100, 1, 1.0)]}
    light = {64: [(c2, 100, 10, 1, 1.0)], 32: [(c2, 100, 10, 1, 1.0)]}

    class Stub:
        def gs_class_variant(self, *a):
            return 0
    monkeypatch.setattr(engine._lib, "lib", lambda: Stub())
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    monkeypatch.setattr(engine, "launch_plan",
                        lambda e, p, kind, cls, *a: (plans if cls == [c1] else light)[p])
    eng = types.SimpleNamespace(segments=[(c1, 0, 100), (c2, 100, 110)], heavy=[(20, 40), (0, 0)])
    cut = lambda: engine.mixed_plan(eng, None, 1e-3)[1]       # noqa: E731
    assert cut() == [(c1, 0, 5, 7, 1), (c1, 5, 95, 6, 1), (c2, 100, 10, 1, 1)]
    eng.heavy_bound = 77
    tiers = cut()
    assert tiers == [(c1, 0, 5, 7, 1, 77), (c1, 5, 35, 6, 1, 77), (c1, 40, 60, 6, 1),
                     (c2, 100, 10, 1, 1)]
    assert engine.launch_records(tiers)["bound"].tolist() == [77, 77, 0, 0]


@pytest.mark.gpu
def test_heavy_quartets_follow_the_largest_density(gpu_lib):
    """Hydrogens in STO-3G: every quartet has 81 primitive quartets, so all are heavy.  With one
    density element of 10 every bound per molecule is above the cut and the build is FP64 (the
    same sums to their order, 1e-14 of elements up to 40); by their own blocks the quartets of the
    other elements, 1e-4, would run in FP32 and be off by 1e-4 x 2^-24 x the sums' magnitude."""
    from gaussium_gb300.batch import BatchedRHF
    from gaussium_gb300.molecules import Molecule
    rng = np.random.default_rng(4)
    grid = np.stack(np.meshgrid([0, 1.4], [0, 1.5], [0, 1.6], indexing="ij"), -1).reshape(-1, 3)
    mols = [Molecule(["H"] * n, grid[:n] + rng.uniform(-0.1, 0.1, (n, 3))) for n in (4, 8, 6)]
    b = BatchedRHF(mols, basis="STO-3G")
    assert all(h[0] == e - s for (_, s, e), h in zip(b.segments, b.heavy))
    packed = []
    for n in (4, 8, 6):
        p = np.full((n, n), 1e-4) * rng.uniform(0.5, 1.0, (n, n))
        p = 0.5 * (p + p.T)
        p[0, 0] = 10.0
        packed.append(p.ravel())
    P = torch.as_tensor(np.concatenate(packed)).to(b.dev)
    full = b.fock_packed(P)
    mixed = b.fock_packed(P, mixed_cut=1e-2, screen_thr=1e-12)
    assert float((mixed - full).abs().max()) <= 1e-13
    # a cut above every bound: FP32
    assert float((b.fock_packed(P, mixed_cut=1e3) - full).abs().max()) > 1e-9
