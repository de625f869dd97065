"""The partition workspace of mixed-precision builds: it never moves while the engine lives,
whatever forms are chosen between two builds, since a captured graph holds its address; each
stream has as much of it as its own longest launch needs."""
import shutil
import types

import numpy as np
import pytest
import torch

from gaussium_gb300 import batch, engine

CLASSES = [(2, 2, 2, 2), (1, 1, 1, 1), (1, 0, 0, 0), (0, 0, 0, 0)]


def read(n, address):
    raw = (engine.ctypes.c_char * (n * engine.LAUNCH_DTYPE.itemsize)).from_address(address)
    return np.frombuffer(bytes(raw), dtype=engine.LAUNCH_DTYPE)


def regions(counts, lanes):
    """Bytes that each of the streams in use needs, launch i on stream i % streams."""
    m = min(len(counts), lanes)
    return [-(-(256 + 16 * int(max(counts[k::m]))) // 256) * 256 for k in range(m)]


class Library:
    """The library calls of a mixed build, without a GPU; ``calls`` keeps the list calls'
    records, workspace address, bytes and stream count."""

    def __init__(self):
        self.forms, self.stamp, self.calls = {}, 0, []

    def choose(self, cls, precision, form):
        self.forms[cls, precision] = form
        self.stamp += 1

    def gs_class_variant_stamp(self):
        return self.stamp

    def gs_class_variant(self, *a):
        return self.forms.get((a[:4], a[4]), 0)

    def gs_class_variants(self, *a):
        return 0b1111111

    def gs_class_form(self, *a):
        return self.gs_class_variant(*a) or engine.WARP_FORM

    def gs_fock_jk_mixed_workspace(self, n):
        return 256 + 16 * n

    def gs_fock_jk_mixed_list_workspace(self, n, list_, lanes):
        return sum(regions(read(n, list_)["count"], lanes))

    def gs_fock_jk_batched(self, *a):
        return 0

    def gs_fock_jk_batched_mixed_list(self, n, list_, *a):
        self.calls.append((read(n, list_), *a[-4:-1]))
        return 0


class Lane:
    def __init__(self, *a):
        pass

    def lane(self, i, *a):
        return None

    def streams(self, lanes):
        return lanes, None

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        pass


@pytest.fixture
def build(monkeypatch):
    """(engine, library, mixed build) of four classes with 50,000 tasks at most."""
    L = Library()
    for m in (batch._lib, engine._lib):
        monkeypatch.setattr(m, "lib", lambda: L)
    monkeypatch.setattr(batch, "HeavyLane", Lane)
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d: types.SimpleNamespace(multi_processor_count=152))
    b = object.__new__(batch.BatchedRHF)
    rng = np.random.default_rng(3)
    b.segments, b.heavy, b.profiles, at = [], [], [], 0
    for cls, n in zip(CLASSES, (300, 20000, 50000, 40000)):
        w = np.sort(rng.integers(1, 40, n))[::-1]
        b.segments.append((cls, at, at + n))
        b.heavy.append(engine.heavy_counts(cls, w))
        b.profiles.append(engine.work_profile(w))
        at += n
    t = torch.zeros(8, dtype=torch.float64)
    b.dev = torch.device("cpu")
    b.tasks = torch.zeros((at, 2), dtype=torch.int32)
    b.pairs = types.SimpleNamespace(rec=t, p64=t, p32=t, prims=lambda p: t)
    b.ds = types.SimpleNamespace(comp_scale=t)
    for name in ("local_fo", "shell_mol", "mol_base", "mol_n", "mol_shell0", "mol_nshell",
                 "mol_sbase"):
        setattr(b, name, t)
    b.block_mol, b.mat_stride = torch.zeros(8, dtype=torch.int64), 8
    b.heavy_bound = 8
    return b, L, lambda cut: b._jk_launch(t, t, t, mixed_cut=cut, dmax=t, screen_thr=1e-12)


def test_workspace_stays_when_forms_change(build):
    b, L, run = build
    run(1e-3)
    first, tiers = b._ws, L.calls[-1][0]
    for cls in CLASSES:
        for p in (64, 32):
            L.choose(cls, p, engine.WARP_FORM)
    run(1e-4)
    assert L.calls[-1][0]["count"].max() > tiers["count"].max()      # another plan
    engine.SPLIT_OFF.update((cls, p) for cls in CLASSES for p in (64, 32))
    run(1e-4)
    assert L.calls[-1][0]["count"].max() == 50000
    assert b._ws is first and len({c[1] for c in L.calls}) == 1
    for records, ws, size, lanes in L.calls:
        assert ws == first.data_ptr() and -size == first.numel() and lanes == engine.MIXED_LANES
        assert sum(regions(records["count"], lanes)) <= first.numel()
    # the longest tier is paid for once
    assert first.numel() <= 16 * b.tasks.shape[0] + 8192


def test_fewer_streams_rather_than_more_memory(build, monkeypatch):
    b, L, run = build
    monkeypatch.setattr(engine, "MIXED_BYTES", 1 << 20)
    run(1e-3)
    records, _, size, lanes = L.calls[-1]
    assert b._ws.numel() == -size == 1 << 20 and 1 < lanes < engine.MIXED_LANES
    assert sum(regions(records["count"], lanes)) <= 1 << 20 < \
        sum(regions(records["count"], lanes + 1))
    monkeypatch.setattr(engine, "MIXED_BYTES", 0)
    del b._ws
    run(1e-3)
    records, _, _, lanes = L.calls[-1]
    assert sum(regions(records["count"], lanes)) <= b._ws.numel() < 16 * 50000 + 1024


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="nvcc not available")
def test_packed_regions_of_a_list():
    """The library's sum of the streams' needs, and its refusal of a workspace below it before
    anything is launched."""
    from gaussium_gb300 import _lib, build
    L = _lib.load_library(build.build())
    counts = [7, 50000, 0, 16, 300, 12, 1]
    records = engine.launch_records([((1, 0, 0, 0), 0, c, 0, 0) for c in counts])
    for lanes in (1, 2, 3, 6, 8, 64):
        need = sum(regions(counts, lanes))
        got = L.gs_fock_jk_mixed_list_workspace(len(records), records.ctypes.data, lanes)
        assert got == need
        streams = (engine.ctypes.c_void_p * lanes)()
        rc = L.gs_fock_jk_mixed_list(len(records), records.ctypes.data, 8, 8, 8, 8, 8, 1, 1, 8, None,
                                     None, 0, None, None, 8, 1e-12, 1e-3, 8, 1 - need, lanes, streams)
        assert rc == 5                                     # GS_ERR_NOMEM
    assert L.gs_fock_jk_mixed_list_workspace(0, None, 6) == 0
    many = np.repeat(records, 16)
    assert L.gs_fock_jk_mixed_list_workspace(len(many), many.ctypes.data, 65) == 0


@pytest.mark.gpu
def test_captured_build_after_forms_change(gpu_lib):
    """A captured mixed build replayed after other forms were chosen and another build ran."""
    from gaussium_gb300 import autotune
    from gaussium_gb300.molecules import water_cluster
    b = batch.BatchedRHF([water_cluster(2, seed=s) for s in range(3)], basis="6-31G*")
    before, _ = b.run(mixed_cut=1e-3, screen_thr=1e-12)
    ws = b._ws
    try:
        for cls, _, _ in b.segments:
            for p in (64, 32):
                if autotune.WARP in autotune.forms(cls, p):
                    autotune.set_form(cls, p, autotune.WARP)
        other, _ = b.run(mixed_cut=1e-4, screen_thr=1e-12)
        again, _ = b.run(mixed_cut=1e-3, screen_thr=1e-12)
    finally:
        autotune.reset(b.segments)
    assert b._ws is ws
    # energies of one final FP64 build each, at densities converged to 1e-10
    assert np.max(np.abs(again - before)) < 1e-8 and np.max(np.abs(other - before)) < 1e-8
