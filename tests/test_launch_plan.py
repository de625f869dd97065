"""Launch plans: the tiers of a class segment, and the cluster form they use for the heaviest
quartets."""
import numpy as np
import pytest
import torch

from gaussium_gb300 import engine

ALL = [(0, 0, 0, 0), (1, 0, 0, 0), (1, 1, 1, 0), (1, 1, 1, 1), (2, 0, 2, 0), (2, 1, 2, 0),
       (2, 1, 1, 1), (2, 2, 2, 1), (2, 2, 2, 2)]


@pytest.mark.parametrize("kind", ["jk", "write"])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("cls", ALL)
def test_tiers_tile_the_segment(cls, precision, kind):
    """Whatever the work, the tiers cover [0, n) once, lightest last; only forms that are built;
    no thread tier where the limit leaves no primitive quartet to it."""
    rng = np.random.default_rng(sum(cls))
    built = 0b1111111 if sum(cls) <= 5 or precision == 32 else 0b1110110
    for n, top, limit in ((1, 1, 600.0), (7, 1296, 600.0), (5000, 40, 600.0), (5000, 1296, 1e5),
                          (300, 0, 600.0), (4096, 200, 1.0)):
        w = np.sort(rng.integers(0, top + 1, n))[::-1]
        plan = engine.class_plan(cls, precision, kind, n, engine.work_profile(w), limit, built)
        at = 0
        for form, first, count, latency in plan:
            assert first == at and count > 0 and latency >= 0
            assert form == 0 or built & (1 << ((form & 255) - 1))
            assert form >> 8 in range(engine.MANY_TASKS + 1)
            at += count
        assert at == n
        forms = [p[0] for p in plan]
        assert len(set(forms)) == len(forms)


def test_segment_profiles_match_host():
    rng = np.random.default_rng(1)
    segs = [np.sort(rng.integers(0, t, n))[::-1] for t, n in ((1300, 500), (1, 3), (200000, 40), (9, 1))]
    bounds = np.concatenate([[0], np.cumsum([len(x) for x in segs])]).tolist()
    cls = [(0, 0, 0, 0), (1, 1, 1, 1), (2, 2, 2, 2), (2, 0, 0, 0)]
    got = engine.segment_profiles(cls, torch.as_tensor(np.concatenate(segs).copy()), bounds)
    for c, w, (heavy, prof) in zip(cls, segs, got):
        assert heavy == engine.heavy_counts(c, w)
        assert prof == engine.work_profile(w)


def test_mixed_plan_tiers(monkeypatch):
    """A segment is cut wherever either precision's form changes, each part in both plans'
    forms; a class whose form was chosen keeps its banded prefix and one partitioned rest."""
    import types
    c1, c2 = (2, 2, 2, 2), (1, 0, 0, 0)
    plans = {64: [(c1, 10, 2, 7, 9.0), (c1, 12, 5, 5, 5.0), (c1, 17, 83, 6, 1.0)],
             32: [(c1, 10, 3, 5, 2.0), (c1, 13, 87, 1, 1.0)]}

    class Stub:
        def gs_class_variant(self, *a):
            return int(a[:4] == c2)

        def gs_class_form(self, *a):
            return engine.THREAD_FORM
    monkeypatch.setattr(engine._lib, "lib", lambda: Stub())
    monkeypatch.setattr(engine, "launch_plan", lambda e, p, *a: plans[p])
    eng = types.SimpleNamespace(segments=[(c1, 10, 100), (c2, 100, 130)], heavy=[(0, 0), (7, 2)])
    banded, tiers = engine.mixed_plan(eng, None, 1e-3)
    assert tiers == [(c1, 10, 2, 7, 5), (c1, 12, 1, 5, 5), (c1, 13, 4, 5, 1), (c1, 17, 83, 6, 1),
                     (c2, 107, 23, 0, 0)]
    inf = float("inf")
    assert banded == [(c2, 100, 64, 4, 7, 1e-3, inf), (c2, 100, 32, 4, 7, 0.0, 1e-3)]
    assert engine.mixed_plan(eng, [c2], 1e-3)[1] == [(c2, 107, 23, 0, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [(64, 1e-13), (32, 1e-5)])
def test_cluster_form_matches_warp_form(gpu_lib, precision, tol):
    """Blocks and J/K of every class built with the cluster form, for quartets of one to 1,296
    primitive quartets (fewer than, and not a multiple of, the cluster's 64 warps)."""
    from gaussium_gb300 import _lib, build
    from gaussium_gb300.basis import ShellBasis
    rng = np.random.default_rng(0)
    shells = []
    for l in range(3):
        for k in (1, 2, 6):
            shells.append(dict(l=l, centre=rng.uniform(-1, 1, 3), expo=np.exp(rng.uniform(-2, 3, k)),
                               coef=rng.uniform(0.2, 1.0, k)))
    sb = ShellBasis.from_shell_dicts(shells)
    eng = engine.JKEngine(sb, schwarz_thr=0.0, max_exp=0.0)
    p = rng.standard_normal((sb.nbf, sb.nbf))
    pt = torch.as_tensor(p + p.T).cuda()
    n = sb.nbf
    seen = 0
    for cls, s, e in eng.segments:
        if not gpu_lib.gs_class_variants(*cls, precision) & 64:
            continue
        seen += 1
        got = {}
        for form in (engine.WARP_FORM, engine.CLUSTER_FORM):
            j = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            k = torch.zeros_like(j)
            rc = gpu_lib.gs_fock_jk(
                *cls, precision | (form << 8), _lib.ptr(eng.pairs.rec),
                _lib.ptr(eng.pairs.prims(precision)), _lib.ptr(eng.ds.comp_scale),
                _lib.ptr(eng.ds.func_off), sb.nshell, n, e - s, eng.tasks.data_ptr() + 8 * s,
                _lib.ptr(pt), _lib.ptr(j), 1, _lib.ptr(pt), _lib.ptr(k), None, 0.0, 0.0, 0.0,
                _lib.stream())
            _lib.check(rc, "gs_fock_jk")
            got[form] = (j, k)
        for x, y in zip(got[engine.WARP_FORM], got[engine.CLUSTER_FORM]):
            assert float((x - y).abs().max()) <= tol * float(x.abs().max()), cls
    assert seen == len([c for c in build.classes() if sum(c) >= 3])
    # the same quartets as blocks, the heavy ones through the plan's cluster tier
    tri = np.array([[a, b, c, d] for a in range(9) for b in range(a + 1) for c in range(9)
                    for d in range(c + 1)])
    batch = engine.QuartetBatch(eng.ds, tri, want32=precision == 32)
    plan = engine.launch_plan(batch, precision, "write")
    assert any(form == engine.CLUSTER_FORM for _, _, _, form, _ in plan)
    out = torch.full((batch.total,), float("nan"), dtype=torch.float64, device="cuda")
    batch.run(out, precision)
    from gaussium_gb300 import autotune
    ref = torch.full_like(out, float("nan"))
    try:
        for cls, _, _ in batch.segments:
            autotune.set_form(cls, precision, autotune.WARP)
            engine.SPLIT_OFF.add((cls, precision))
        batch.run(ref, precision)
    finally:
        autotune.reset(batch.segments)
    assert float((out - ref).abs().max()) <= tol * float(ref.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_many_quartets_a_warp(gpu_lib, precision):
    """Blocks are the same bits with one to eight quartets a warp, J/K the same sums up to the
    atomics' order: tasks of zero (screened out) to 36 primitive quartets, counts that are no
    multiple of the warp's, screened tasks among them."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.workloads import random_shell_quartets
    sb, _, _ = random_shell_quartets(8, seed=11, box_angstrom=6.0, kmax=3)
    ns = sb.nshell
    q = np.random.default_rng(4).integers(0, ns, (3001, 4))
    ds = engine.DeviceShells(sb)
    batch = engine.QuartetBatch(ds, q, want32=True, max_exp=engine.PRIM_SCREEN)
    assert any(prof[1][0] < e - s for (_, s, e), prof in zip(batch.segments, batch.profiles))
    eng = engine.JKEngine(sb, schwarz_thr=0.0, max_exp=engine.PRIM_SCREEN)
    n = sb.nbf
    p = np.random.default_rng(5).standard_normal((n, n))
    pt = torch.as_tensor(p + p.T).cuda()
    dmax = eng.shell_dmax([pt])
    for form in (engine.WARP_FORM, engine.GROUPED_FORM, engine.STACKED_FORM):
        ref = None
        for per in (0, 1, 2, 5, 8):
            out = torch.full((batch.total,), float("nan"), dtype=torch.float64, device="cuda")
            j = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            k = torch.zeros_like(j)
            for cls, s, e in batch.segments:
                f = form if gpu_lib.gs_class_variants(*cls, precision) & (1 << (form - 1)) else \
                    engine.WARP_FORM
                _lib.check(gpu_lib.gs_eri_blocks(
                    *cls, precision | f << 8 | per << 16, _lib.ptr(batch.pairs.rec),
                    _lib.ptr(batch.pairs.prims(precision)), _lib.ptr(ds.comp_scale), e - s,
                    batch.tasks.data_ptr() + s * engine.WRITE_TASK, _lib.ptr(out),
                    _lib.stream()), "gs_eri_blocks")
            for cls, s, e in eng.segments:
                f = form if gpu_lib.gs_class_variants(*cls, precision) & (1 << (form - 1)) else \
                    engine.WARP_FORM
                _lib.check(gpu_lib.gs_fock_jk(
                    *cls, precision | f << 8 | per << 16, _lib.ptr(eng.pairs.rec),
                    _lib.ptr(eng.pairs.prims(precision)), _lib.ptr(eng.ds.comp_scale),
                    _lib.ptr(eng.ds.func_off), ns, n, e - s, eng.tasks.data_ptr() + 8 * s,
                    _lib.ptr(pt), _lib.ptr(j), 1, _lib.ptr(pt), _lib.ptr(k), _lib.ptr(dmax), 1e-6,
                    1e-5, float("inf"), _lib.stream()), "gs_fock_jk")
            got = (out, j, k)
            if ref is None:
                ref = got
                assert not bool(torch.isnan(out).any())
            assert torch.equal(out, ref[0]), (form, per)
            for x, y in zip(got[1:], ref[1:]):
                assert float((x - y).abs().max()) <= 1e-13 * float(y.abs().max())
    assert gpu_lib.gs_eri_blocks(0, 0, 0, 0, precision | 2 << 8 | 9 << 16, _lib.ptr(batch.pairs.rec),
                                 _lib.ptr(batch.pairs.p64), _lib.ptr(ds.comp_scale), 0, None,
                                 _lib.ptr(ref[0]), None) == 1


@pytest.mark.gpu
def test_gradient_tasks_a_warp(gpu_lib):
    """The warp form of the adjoint with one to eight quartets a warp, screened ones among
    them: the same gradient up to the atomics' order."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.molecules import shell_basis, water_cluster
    mol = water_cluster(2, seed=1)
    sb = shell_basis(mol, "6-31G*")
    eng = engine.JKEngine(sb, schwarz_thr=1e-12)
    from gaussium_gb300.gradient import shell_atoms
    sa = torch.as_tensor(shell_atoms(mol, sb).astype(np.int32)).cuda()
    p = np.random.default_rng(2).standard_normal((sb.nbf, sb.nbf)) * 0.1
    pt = torch.as_tensor(p + p.T).cuda()
    dmax = eng.shell_dmax([pt])
    ref = None
    for per in (0, 1, 3, 8):
        g = torch.zeros(18, dtype=torch.float64, device="cuda")
        for cls, s, e in eng.segments:
            _lib.check(gpu_lib.gs_eri_grad_band(
                *cls, 2 | per << 8, 64, _lib.ptr(eng.pairs.rec), _lib.ptr(eng.pairs.p64),
                _lib.ptr(eng.ds.comp_scale), _lib.ptr(eng.ds.func_off), _lib.ptr(sa), e - s,
                eng.tasks.data_ptr() + 8 * s, sb.nbf, 6, _lib.ptr(pt), sb.nshell, _lib.ptr(dmax),
                1e-7, 0.0, float("inf"), _lib.ptr(g), _lib.stream()), "gs_eri_grad_band")
        ref = g if ref is None else ref
        assert float((g - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    assert abs(float(g.view(6, 3).sum())) < 1e-10          # translational invariance


@pytest.mark.gpu
@pytest.mark.parametrize("form", [1, 3])
def test_gradient_partition_matches_bands(gpu_lib, form):
    """The partitioned adjoint evaluates the quartets of the two bands, each in its precision:
    the same gradient up to the order of the sums."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.gradient import shell_atoms
    from gaussium_gb300.molecules import shell_basis, water_cluster
    mol = water_cluster(2, seed=2)
    sb = shell_basis(mol, "6-31G*")
    eng = engine.JKEngine(sb, schwarz_thr=1e-12)
    sa = torch.as_tensor(shell_atoms(mol, sb).astype(np.int32)).cuda()
    p = np.random.default_rng(3).standard_normal((sb.nbf, sb.nbf)) * 0.1
    pt = torch.as_tensor(p + p.T).cuda()
    dmax = eng.shell_dmax([pt])
    ws = torch.empty(gpu_lib.gs_fock_jk_mixed_workspace(eng.ntasks), dtype=torch.uint8, device="cuda")
    inf = float("inf")
    for cls, s, e in eng.segments:
        if sum(cls) > 3:
            continue
        tail = (_lib.ptr(eng.ds.comp_scale), _lib.ptr(eng.ds.func_off), _lib.ptr(sa), e - s,
                eng.tasks.data_ptr() + 8 * s, sb.nbf, 6, _lib.ptr(pt), sb.nshell, _lib.ptr(dmax))
        a, b = (torch.zeros(18, dtype=torch.float64, device="cuda") for _ in range(2))
        for prec, prims, lo, hi in ((64, eng.pairs.p64, 1e-3, inf), (32, eng.pairs.p32, 0.0, 1e-3)):
            _lib.check(gpu_lib.gs_eri_grad_band(
                *cls, form, prec, _lib.ptr(eng.pairs.rec), _lib.ptr(prims), *tail, 1e-9, lo, hi,
                _lib.ptr(a), _lib.stream()), "gs_eri_grad_band")
        call = (*cls, form, _lib.ptr(eng.pairs.rec), _lib.ptr(eng.pairs.p64),
                _lib.ptr(eng.pairs.p32), *tail, 1e-9, 1e-3, _lib.ptr(b), _lib.ptr(ws))
        _lib.check(gpu_lib.gs_eri_grad_mixed(*call, ws.numel(), _lib.stream()), "gs_eri_grad_mixed")
        assert float((a - b).abs().max()) <= 1e-12 * float(a.abs().max()), cls
        assert gpu_lib.gs_eri_grad_mixed(*call, 256, None) == 5


@pytest.mark.gpu
def test_task_keys(gpu_lib):
    """Key fields against their definition: counts exactly, the distance bin to a rounding."""
    from gaussium_gb300.workloads import random_shell_quartets
    sb, _, _ = random_shell_quartets(4, seed=9, box_angstrom=8.0)
    eng = engine.JKEngine(sb, schwarz_thr=0.0)
    n = eng.npairs
    rng = np.random.default_rng(0)
    bra, ket = (torch.as_tensor(rng.integers(0, n, 4000)).cuda() for _ in range(2))
    keys = engine.task_keys(eng.pairs, bra, ket).cpu().numpy()
    b, k = bra.cpu().numpy(), ket.cpu().numpy()
    nprim = eng.pairs.nprim
    assert np.array_equal(keys >> 6, nprim[b] * nprim[k] * 4096 + nprim[b] * 64 + nprim[k])
    assert np.array_equal(keys // engine.KEY_WORK, nprim[b] * nprim[k])
    rec = eng.pairs.p64.cpu().numpy().view(np.float64).reshape(-1, 10)
    at = eng.pairs.prim_start.cpu().numpy() + np.maximum(nprim - 1, 0)
    d2 = ((rec[at[b], 2:5] - rec[at[k], 2:5]) ** 2).sum(1) + 0.25
    want = np.where(nprim[b] * nprim[k] > 0, np.clip(np.floor(2 * np.log2(d2)) + 4, 0, 63), 0)
    both = np.abs((keys & 63) - want)
    assert both.max() <= 1          # steps are sqrt(2) or 3/2 and 4/3: not quite the logarithm's
    assert np.mean(both) < 0.2


@pytest.mark.parametrize("seed", range(4))
def test_unique_pair_ranges(seed):
    """The ranges hold every unique pair of pairs once, bra class >= ket class, and each class
    segment is one run of them by descending primitive-quartet count."""
    rng = np.random.default_rng(seed)
    n = [1, 7, 40, 91][seed]
    pc = np.sort(rng.integers(0, 6, n))
    npp = rng.choice([1, 3, 6, 9, 18, 36], n)
    order = np.lexsort((-npp, pc))
    pc, npp = pc[order], npp[order]
    ranges, work, segs = engine.unique_pair_ranges(pc, npp)
    seen, at = set(), 0
    for r, (w, count) in zip(ranges, work):
        assert r["first"] == at
        at += count
        b = range(r["bra"], r["bra"] + r["nbra"])
        mine = [(x, y) for x in b for y in range(r["ket"], r["ket"] + r["nket"])] if r["nket"] else \
            [(x, y) for x in b for y in range(r["bra"], x + 1)]
        assert len(mine) == count
        for x, y in mine:
            assert pc[x] >= pc[y] and npp[x] * npp[y] == w
            assert (max(x, y), min(x, y)) not in seen
            seen.add((max(x, y), min(x, y)))
    assert len(seen) == n * (n + 1) // 2 == at == segs[-1][2]
    for cls, s, e in segs:
        w = [x[0] for r, x in zip(ranges, work) if s <= r["first"] < e]
        assert w == sorted(w, reverse=True)


@pytest.mark.gpu
@pytest.mark.parametrize("basis,waters", [("STO-3G", 1), ("6-31G*", 2)])
def test_dense_tensor_from_ranges(gpu_lib, basis, waters, monkeypatch):
    """The dense tensor from pair ranges against the one from a host list of quartets."""
    from gaussium_gb300 import dropin
    from gaussium_gb300.molecules import shell_basis, water_cluster
    sb = shell_basis(water_cluster(waters, seed=3), basis)
    a = dropin.dense_eri(sb)
    monkeypatch.setattr(engine, "MAX_RANGES", 0)
    b = dropin.dense_eri(sb)
    assert float((a - b).abs().max()) <= 1e-14 * float(b.abs().max())
    for perm in ((1, 0, 2, 3), (0, 1, 3, 2), (2, 3, 0, 1)):
        assert torch.equal(a, a.permute(perm))


def test_upload_views():
    arrays = [np.arange(5, dtype=np.int32), np.zeros((0, 2), np.float64), np.ones((3, 2)),
              np.arange(3, dtype=np.int64)]
    got = engine.upload("cpu", *arrays)
    for a, t in zip(arrays, got):
        assert t.numpy().dtype == a.dtype and np.array_equal(t.numpy(), a)
        assert t.data_ptr() % 8 == 0


@pytest.mark.gpu
def test_mixed_forms_match(gpu_lib):
    """The partitioned launch gives the same J/K in every pair of forms, the heavy forms with
    their counts on the device among them; an unknown form is refused."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.workloads import random_shell_quartets
    sb, _, _ = random_shell_quartets(4, seed=5, box_angstrom=3.0, kmax=4)
    eng = engine.JKEngine(sb, schwarz_thr=0.0)
    n = sb.nbf
    p = np.random.default_rng(6).standard_normal((n, n))
    pt = torch.as_tensor(p + p.T).cuda()
    dmax = eng.shell_dmax([pt])
    ws = torch.empty(gpu_lib.gs_fock_jk_mixed_workspace(eng.ntasks), dtype=torch.uint8, device="cuda")
    for cls, s, e in eng.segments:
        forms = {q: [f for f in range(1, 8) if gpu_lib.gs_class_variants(*cls, q) & (1 << (f - 1))]
                 for q in (64, 32)}
        ref = None
        for i in range(max(len(x) for x in forms.values())):
            f64, f32 = (x[i % len(x)] for x in forms.values())
            j = torch.zeros((n, n), dtype=torch.float64, device="cuda")
            k = torch.zeros_like(j)

            def call(f64, f32):
                return gpu_lib.gs_fock_jk_mixed_forms(
                    *cls, f64, f32, _lib.ptr(eng.pairs.rec), _lib.ptr(eng.pairs.p64),
                    _lib.ptr(eng.pairs.p32), _lib.ptr(eng.ds.comp_scale),
                    _lib.ptr(eng.ds.func_off), sb.nshell, n, e - s, eng.tasks.data_ptr() + 8 * s,
                    _lib.ptr(pt), _lib.ptr(j), 1, _lib.ptr(pt), _lib.ptr(k), _lib.ptr(dmax), 1e-12,
                    1e-4, _lib.ptr(ws), ws.numel(), _lib.stream())
            _lib.check(call(f64, f32), "gs_fock_jk_mixed_forms")
            ref = (j, k) if ref is None else ref
            # FP32 quartets are below 1e-4: their rounding, 1e-5 of it, on up to 1e4 of them
            for x, y in zip((j, k), ref):
                assert float((x - y).abs().max()) <= 1e-5 * 1e-4 * 1e4 * 1e-2 + \
                    1e-12 * float(y.abs().max()), (cls, f64, f32)
            assert call(8, 0) == 1 and call(0, -1) == 1


def test_kept_plans_follow_the_forms(monkeypatch):
    """A kept plan is built again once a class's form is chosen, a class leaves or joins
    SPLIT_OFF, or the precision cut changes, and only then; records have the C ABI's layout."""
    stamp, built = [0], []

    class Stub:
        def gs_class_variant_stamp(self):
            return stamp[0]

    class Eng:
        pass

    monkeypatch.setattr(engine._lib, "lib", lambda: Stub())
    monkeypatch.setattr(engine, "SPLIT_OFF", set())
    plan = [((2, 1, 1, 0), 1 << 40, 7, 5 | 3 << 8, 2)]
    monkeypatch.setattr(engine, "mixed_plan", lambda e, c, cut: (built.append(cut) or [], plan))
    eng = Eng()
    get = lambda cut: engine.mixed_list(eng, None, cut)[1]      # noqa: E731
    r = get(1e-3)
    assert engine.LAUNCH_DTYPE.itemsize == 40 and r.tobytes() == np.array(
        [2, 1, 1, 0, 5 | 3 << 8, 2, 7, 0, 0, 1 << 8], dtype="<i4").tobytes()
    assert get(1e-3) is r and len(built) == 1
    stamp[0] += 1
    assert get(1e-3) is not r and len(built) == 2
    engine.SPLIT_OFF.add(((1, 0, 0, 0), 64))
    get(1e-3), get(1e-3)
    assert len(built) == 3
    get(1e-4), get(1e-4)
    assert built == [1e-3, 1e-3, 1e-3, 1e-4]


@pytest.mark.gpu
@pytest.mark.parametrize("nstreams", [1, 3, 8])
def test_list_calls_match_single_launches(gpu_lib, nstreams):
    """A list of launches over several streams gives what the launches one by one give (sums in
    another order: 1e-13 of the largest element); no launch is an empty list; a class that is not
    built, a negative form and a missing stream array are refused, and what ran before is joined."""
    import ctypes
    from gaussium_gb300 import _lib
    from gaussium_gb300.workloads import random_shell_quartets
    sb, _, _ = random_shell_quartets(4, seed=5, box_angstrom=3.0, kmax=4)
    eng = engine.JKEngine(sb, schwarz_thr=0.0)
    n = sb.nbf
    p = np.random.default_rng(9).standard_normal((n, n))
    pt = torch.as_tensor(p + p.T).cuda()
    dmax = eng.shell_dmax([pt])
    plan = engine.launch_list(eng, 64, "jk")
    sides = [torch.cuda.Stream() for _ in range(nstreams - 1)]
    handles = (ctypes.c_void_p * nstreams)(*[x.cuda_stream for x in sides],
                                           torch.cuda.current_stream().cuda_stream)

    def fock(records, streams=handles, count=nstreams):
        j = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        k = torch.zeros_like(j)
        rc = gpu_lib.gs_fock_jk_list(
            len(records), records.ctypes.data, 64, _lib.ptr(eng.pairs.rec), _lib.ptr(eng.pairs.p64),
            _lib.ptr(eng.ds.comp_scale), _lib.ptr(eng.ds.func_off), sb.nshell, n,
            eng.tasks.data_ptr(), _lib.ptr(pt), _lib.ptr(j), 1, _lib.ptr(pt), _lib.ptr(k),
            _lib.ptr(dmax), 1e-12, 0.0, float("inf"), count, streams)
        return rc, j, k

    parts = [fock(plan[i:i + 1]) for i in range(len(plan))]
    assert len(plan) > 8 and all(rc == 0 for rc, _, _ in parts)
    rc, j, k = fock(plan)
    assert rc == 0
    for i, x in ((1, j), (2, k)):
        ref = sum(part[i] for part in parts)
        assert float((x - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
    rc, j, k = fock(plan[:0])
    assert rc == 0 and not j.any() and not k.any()
    bad = plan[:3].copy()
    bad["form"][2] = -1
    rc, j, _ = fock(bad)
    assert rc == 1 and not j.any()
    assert fock(plan, None)[0] == 1 and fock(plan, handles, 0)[0] == 1
    bad = plan[:3].copy()
    bad["cls"][2] = (3, 3, 3, 3)
    rc, j, _ = fock(bad)
    ref = parts[0][1] + parts[1][1]
    assert rc == 3 and float((j - ref).abs().max()) <= 1e-13 * float(ref.abs().max())
    # blocks: each has one writer, so the values are the same bit for bit
    sb, quartets, _ = random_shell_quartets(300, seed=8, box_angstrom=3.0, kmax=3)
    b = engine.QuartetBatch(engine.DeviceShells(sb, "cuda"), quartets)
    recs = engine.launch_list(b, 64, "write")
    outs = [torch.zeros(b.total, dtype=torch.float64, device="cuda") for _ in range(2)]
    for r, out in ([(recs, outs[0])] + [(recs[i:i + 1], outs[1]) for i in range(len(recs))]):
        _lib.check(gpu_lib.gs_eri_blocks_list(
            len(r), r.ctypes.data, 64, _lib.ptr(b.pairs.rec), _lib.ptr(b.pairs.p64),
            _lib.ptr(b.ds.comp_scale), b.tasks.data_ptr(), _lib.ptr(out), nstreams, handles),
            "gs_eri_blocks_list")
    assert torch.equal(*outs)


@pytest.mark.gpu
@pytest.mark.parametrize("thr,cut", [(1e-12, 1e-3), (1e-300, 1e-4), (0.25, 0.25), (3e-13, float("inf")),
                                     (0.0, 0.0)])
def test_partition_decides_as_the_double_bound(gpu_lib, thr, cut):
    """The lists of a partition are those of the bound in double, for bounds at, one step beside
    and far from either limit, and too small or large for float."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.workloads import random_shell_quartets
    sb, _, _ = random_shell_quartets(4, seed=5, box_angstrom=3.0, kmax=2)
    eng = engine.JKEngine(sb, schwarz_thr=0.0)
    rng = np.random.default_rng(11)
    n, ns = sb.nbf, sb.nshell
    rec = np.frombuffer(eng.pairs.rec.cpu().numpy().tobytes(), dtype=np.dtype(
        [("ab", "<f8", 3), ("i", "<i4", 4), ("q", "<f4"), ("pad", "<i4")])).copy()
    rec["q"] = 2.0 ** rng.integers(-3, 3, len(rec))
    rec["q"][:4] = 0.0, 1e-38, 3e38, 1e-20
    eng.pairs.rec.copy_(torch.as_tensor(np.frombuffer(rec.tobytes(), dtype=np.uint8).copy()))
    near = [x for x in (thr, cut) if 0.0 < x < 1e30] or [1.0]
    near = np.array([f(x * 2.0 ** k) for x in near for k in range(-6, 7) for f in
                     (lambda y: y, lambda y: np.nextafter(y, 0), lambda y: np.nextafter(y, 9),
                      lambda y: y * (1 + 1e-7), lambda y: y * (1 - 3e-7))])
    d = near[rng.integers(0, len(near), (ns, ns))]
    d[rng.random((ns, ns)) < 0.05] = 0.0
    d[rng.random((ns, ns)) < 0.5] *= 1e-9            # so that the largest of six varies
    dmax = torch.as_tensor(np.maximum(d, d.T)).cuda()
    d = dmax.cpu().numpy()
    pt = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    tasks = eng.tasks[:eng.ntasks].cpu().numpy()
    seen = set()
    for cls, s, e in eng.segments:
        j, k = torch.zeros_like(pt), torch.zeros_like(pt)
        ws = torch.zeros(gpu_lib.gs_fock_jk_mixed_workspace(e - s), dtype=torch.uint8, device="cuda")
        _lib.check(gpu_lib.gs_fock_jk_mixed(
            *cls, _lib.ptr(eng.pairs.rec), _lib.ptr(eng.pairs.p64), _lib.ptr(eng.pairs.p32),
            _lib.ptr(eng.ds.comp_scale), _lib.ptr(eng.ds.func_off), ns, n, e - s,
            eng.tasks.data_ptr() + 8 * s, _lib.ptr(pt), _lib.ptr(j), 1, _lib.ptr(pt), _lib.ptr(k),
            _lib.ptr(dmax), thr, cut, _lib.ptr(ws), ws.numel(), _lib.stream()), "gs_fock_jk_mixed")
        raw = np.frombuffer(ws.cpu().numpy().tobytes(), dtype="<i4")
        t = tasks[s:e]
        B, K = rec[t[:, 0]], rec[t[:, 1]]
        (a, b), (c, f) = B["i"][:, 2:].T, K["i"][:, 2:].T
        dm = np.max([d[a, b], d[c, f], d[a, c], d[a, f], d[b, c], d[b, f]], axis=0)
        est = B["q"].astype(float) * K["q"].astype(float) * dm
        kind = np.where(est < thr, 0, np.where(est >= cut, 1, 2))
        lists = raw[64:64 + 2 * (e - s)], raw[64 + 2 * (e - s):64 + 4 * (e - s)]
        for which in (1, 2):
            got = lists[which - 1].reshape(-1, 2)[:raw[which - 1]]
            assert sorted(map(tuple, got.tolist())) == sorted(map(tuple, t[kind == which].tolist()))
        seen |= set(kind.tolist())
    assert len(seen) >= (1 if thr == cut == 0.0 else 2)
