"""Side streams join the caller's also where a launch between fork and join raises: the buffers
that run on them go back to the caller's stream's allocator."""
import types

import numpy as np
import pytest
import torch

from gaussium_gb300 import _lib, batch, engine, gradient


class Recorder:
    """A HeavyLane whose fork and join are only recorded."""
    log = []

    def __init__(self, *a):
        self.main = types.SimpleNamespace(wait_stream=lambda s: self.log.append(("join", s)))
        self.sides, self.forked = list(range(engine.SIDE_STREAMS)), [False] * engine.SIDE_STREAMS

    def stream(self, k=0):
        self.forked[k] = True
        self.log.append(("fork", k))

    def lane(self, i, lanes=engine.SIDE_STREAMS + 1):
        i %= lanes
        return None if i == lanes - 1 else self.stream(i)

    def streams(self, lanes):
        return lanes, None

    __enter__, __exit__ = engine.HeavyLane.__enter__, engine.HeavyLane.__exit__
    join = engine.HeavyLane.join


@pytest.fixture(autouse=True)
def recorder(monkeypatch):
    monkeypatch.setattr(Recorder, "log", [])
    for m in (batch, engine, gradient):
        monkeypatch.setattr(m, "HeavyLane", Recorder)
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d: types.SimpleNamespace(multi_processor_count=152))


class Failing:
    """A library whose calls return an error from the ``after``-th launch on."""

    def __init__(self, after):
        self.left = after

    def gs_status_string(self, rc):
        return b"planned"

    def gs_fock_jk_mixed_workspace(self, n):
        return 256 + 16 * n

    def gs_eri_grad_class_form(self, *a):
        return 1

    def launch(self, *a):
        self.left -= 1
        return int(self.left < 0)

    gs_fock_jk = gs_fock_jk_batched = gs_eri_grad_mixed = gs_eri_grad_band = launch

    def gs_fock_jk_mixed_list_workspace(self, *a):
        return 0

    def gs_fock_jk_mixed_list(self, *a):
        return 1

    gs_fock_jk_batched_mixed_list = gs_fock_jk_mixed_list


def engine_like(kind):
    t = torch.zeros((2, 2), dtype=torch.float64)
    e = object.__new__(kind)
    e.dev = torch.device("cpu")
    e.segments, e.heavy = [((1, 0, 0, 0), 0, 40), ((0, 0, 0, 0), 40, 80)], [(10, 5), (20, 10)]
    e.profiles = [engine.work_profile(np.full(40, 2))] * 2
    e.tasks = torch.zeros((80, 2), dtype=torch.int32)
    e.pairs = types.SimpleNamespace(rec=t, p64=t, p32=t, prims=lambda p: t)
    e.ds = types.SimpleNamespace(comp_scale=t, func_off=t)
    return e, t


def joined():
    forks = {k for what, k in Recorder.log if what == "fork"}
    assert forks and {k for what, k in Recorder.log if what == "join"} == forks
    assert Recorder.log[-1][0] == "join"


@pytest.mark.parametrize("after", [1, 100])
def test_mixed_builds(monkeypatch, after):
    L = Failing(after)
    for m in (batch, engine, gradient):
        monkeypatch.setattr(m._lib, "lib", lambda: L)
    banded = [((1, 0, 0, 0), 0, 64, 4, 10, 0.0, 1.0)] * 3
    none = engine.launch_records([])
    for m in (batch, engine):
        monkeypatch.setattr(m, "mixed_list", lambda *a: (banded, none))
    b, t = engine_like(batch.BatchedRHF)
    for name in ("local_fo", "shell_mol", "mol_base", "mol_n", "mol_shell0", "mol_nshell", "mol_sbase"):
        setattr(b, name, t)
    b.block_mol, b.mat_stride, b.heavy_bound = torch.zeros(4, dtype=torch.int64), 4, 4
    with pytest.raises(_lib.GsError):
        b._jk_launch(t, t, t, mixed_cut=1e-3, dmax=torch.zeros(4, dtype=torch.float64))
    joined()
    Recorder.log.clear()
    e, t = engine_like(engine.JKEngine)
    e.sb, e.shell_dmax = types.SimpleNamespace(nbf=2, nshell=2), lambda mats: t
    monkeypatch.setattr(engine, "_check_device_tensor", lambda *a: None)
    with pytest.raises(_lib.GsError):
        e.jk(t, [t], mixed_cut=1e-3)
    joined()


def test_gradient(monkeypatch):
    L = Failing(2)
    monkeypatch.setattr(gradient._lib, "lib", lambda: L)
    monkeypatch.setattr(gradient, "_check_atoms", lambda *a: None, raising=False)
    e, t = engine_like(engine.JKEngine)
    e.shell_dmax = lambda mats: t
    sb = types.SimpleNamespace(nbf=2, nshell=2)
    with pytest.raises(_lib.GsError):
        gradient.eri_gradient(sb, e, np.zeros(2, dtype=np.int32), np.zeros((2, 2)), 1)
    joined()
    # the one-electron kernel's stream too, whatever the adjoint raises
    Recorder.log.clear()

    def one(ds, mol, sa, P, W, lane):
        return torch.zeros(3), (lane.stream(engine.SIDE_STREAMS - 1),)

    def adjoint(*a, **kw):
        raise MemoryError
    monkeypatch.setattr(gradient, "_one_electron_launch", one)
    monkeypatch.setattr(gradient, "eri_gradient", adjoint)
    monkeypatch.setattr(gradient, "shell_atoms", lambda mol, sb: np.zeros(2, dtype=np.int32))
    mol = types.SimpleNamespace(symbols=["H"])
    with pytest.raises(MemoryError):
        gradient.gradient_from_state(gradient.RHFState(mol, sb, e, 0.0, None, None, None))
    joined()
