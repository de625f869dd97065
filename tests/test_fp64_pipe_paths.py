"""The paths that keep work off the FP64 pipe: the FP32 Boys function in float pairs, the
integer conversions of the Fock digestion, and blocks of unit component scales."""
import numpy as np
import pytest
import torch

import hostcheck
import oracle
from gaussium_gb300 import autotune, engine
from gaussium_gb300.basis import ShellBasis
from gaussium_gb300.workloads import random_shell_quartets

ASYM32 = [17, 20, 23, 25, 28, 30, 32, 34, 36, 38]


@pytest.mark.parametrize("m", range(10))
def test_boys_pair32_rounds_like_fp64(m):
    """One float rounding (2^-24 relative), plus three float roundings each of the two
    expansions' remainders, which are at most 1/32 of the leading terms: 1.25 x 2^-24."""
    L = hostcheck.hc()
    rng = np.random.default_rng(m)
    t = np.concatenate([[0.0, 1 / 32, 1 / 16, 3 / 32, np.nextafter(ASYM32[m], 0)],
                        np.exp(rng.uniform(np.log(1e-4), np.log(ASYM32[m]), 300))])
    t = t.astype(np.float32).astype(np.float64)
    t = t[t < ASYM32[m]]
    F = np.zeros(m + 1)
    for x in t:
        assert L.hc_boys_pair32(m, float(x), F.ctypes.data) == 0
        ex = np.array([oracle.boys_exact(k, float(x)) for k in range(m + 1)])
        assert np.max(np.abs(F / ex - 1.0)) < 1.25 * 2.0 ** -24, x


ASYM64 = [36, 40, 43, 46, 49, 52, 54, 57, 59, 61, 64]


@pytest.mark.parametrize("m", range(11))
def test_boys_row64(m):
    """The expansions' error (2^-52.6 from the float terms, 2^-54 from the terms left out, a
    rounding of 2^-53 at each of two multiply-adds of full size) and 2^-53 for each of the two
    operations an order of the downward recursion: (4 + 2 m) 2^-53, as much again for the
    reference's own rounding."""
    L = hostcheck.hc()
    rng = np.random.default_rng(m)
    t = np.concatenate([[0.0, 1 / 64, 1 / 32, 3 / 64, np.nextafter(1 / 64, 1), np.nextafter(ASYM64[m], 0)],
                        np.exp(rng.uniform(np.log(1e-6), np.log(ASYM64[m]), 400)),
                        rng.uniform(0, ASYM64[m], 400)])
    F = np.zeros(m + 1)
    for x in t:
        assert L.hc_boys_row64(m, float(x), F.ctypes.data) == 0
        ex = np.array([oracle.boys_exact(k, float(x)) for k in range(m + 1)])
        assert np.max(np.abs(F / ex - 1.0)) < 2 * (4 + 2 * m) * 2.0 ** -53, x


def _small_basis(seed, scales):
    sb, _, _ = random_shell_quartets(3, seed=seed, box_angstrom=1.5, lmax=1)
    cs = np.random.default_rng(seed).uniform(0.5, 2.0, (sb.nshell, 6)) if scales else \
        np.ones((sb.nshell, 6))
    return ShellBasis(sb.l, sb.centre, sb.prim_off, sb.expo, sb.coef, cs)


@pytest.mark.gpu
@pytest.mark.parametrize("form", [autotune.THREAD, autotune.WARP])
def test_component_scales(gpu_lib, form):
    """Scaled components give the unit-scale result times the scales: J of the scaled basis
    is s J[s P s] s of the unit one, a few roundings apart."""
    unit, scaled = _small_basis(3, False), _small_basis(3, True)
    s = np.concatenate([scaled.comp_scale[i, :n] for i, n in enumerate(scaled.nfunc)])
    p = np.random.default_rng(0).standard_normal((unit.nbf, unit.nbf))
    p = p + p.T
    a, b = engine.JKEngine(unit, schwarz_thr=0.0), engine.JKEngine(scaled, schwarz_thr=0.0)
    d = lambda x: torch.as_tensor(x).cuda()   # noqa: E731
    try:
        for cls, _, _ in a.segments:
            if form in autotune.forms(cls, 64):
                autotune.set_form(cls, 64, form)
        ja, (ka,) = a.jk(d(s[:, None] * p * s), [d(s[:, None] * p * s)])
        jb, (kb,) = b.jk(d(p), [d(p)])
    finally:
        autotune.reset(a.segments)
    ss = d(np.outer(s, s))
    for x, y in ((ja, jb), (ka, kb)):
        assert float((x * ss - y).abs().max()) < 1e-13 * float(y.abs().max())


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [1.0, 1e-20, 1e-45, 0.0, 1e30])
def test_fp32_digestion_of_any_density(gpu_lib, scale):
    """The FP32 digestion's conversions over the floats' range, their subnormals and zero:
    FP32 J and K are the FP64 ones to FP32 accuracy (1e-5 of the largest); among subnormals
    each of the about 600 terms of a sum is off by the smallest float (1.4e-45) times an
    integral of at most about 10."""
    sb = _small_basis(5, False)
    eng = engine.JKEngine(sb, schwarz_thr=0.0)
    p = np.random.default_rng(1).standard_normal((sb.nbf, sb.nbf))
    p = (p + p.T) * scale
    p[0, :] = p[:, 0] = 0.0
    pt = torch.as_tensor(p).cuda()
    j64, (k64,) = eng.jk(pt, [pt], precision=64)
    j32, (k32,) = eng.jk(pt, [pt], precision=32)
    for x, y in ((j64, j32), (k64, k32)):
        tol = 1e-5 * float(x.abs().max()) + 1e-41
        assert float((x - y).abs().max()) <= tol


@pytest.mark.gpu
def test_rsqrt(gpu_lib):
    """Two units in the last place (the step's error under 2^-58 and five roundings) from the
    smallest to the largest normal number; the library's values outside."""
    from gaussium_gb300 import _lib
    rng = np.random.default_rng(3)
    x = np.concatenate([np.exp(rng.uniform(np.log(2.3e-308), np.log(1.7e308), 200000)),
                        rng.uniform(1.0, 4.0, 200000),
                        [2.2250738585072014e-308, 1.7976931348623157e308, 1.0, 2.0, 4.0]])
    d = torch.as_tensor(x).cuda()
    y = torch.empty_like(d)
    _lib.check(gpu_lib.gs_rsqrt_eval(len(x), _lib.ptr(d), _lib.ptr(y), _lib.stream()), "rsqrt")
    exact = 1.0 / np.sqrt(x.astype(np.longdouble))
    assert float(np.max(np.abs(y.cpu().numpy() / exact - 1.0))) <= 2 * 2.0 ** -52
    odd = torch.tensor([0.0, -0.0, 5e-324, 1e-310, float("inf"), float("nan"), -1.0],
                       dtype=torch.float64, device="cuda")
    got = torch.empty_like(odd)
    _lib.check(gpu_lib.gs_rsqrt_eval(7, _lib.ptr(odd), _lib.ptr(got), _lib.stream()), "rsqrt")
    assert torch.allclose(got, torch.rsqrt(odd), rtol=1e-15, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("max_exp", [0.0, 55.0, 3.0])
@pytest.mark.parametrize("count", [False, True])
def test_pair_records_against_extended_precision(gpu_lib, max_exp, count):
    """Primitive-pair records of exponents over 17 decades and centres on, near and far from each
    other: p exact, 1/2p to 1 ulp, P - A = -b/p AB to five roundings, P to one more, the Gaussian
    product prefactor to ten roundings and ten of its exponent; the kept
    pairs are those of the screen's double-precision test, in both kernels."""
    from gaussium_gb300 import _lib
    rng = np.random.default_rng(3)
    shells = []
    for i in range(24):
        c = rng.standard_normal(3) * (0.0, 1e-9, 0.3, 2.0, 40.0)[i % 5]
        k = (1, 3, 6)[i % 3]
        expo = 10.0 ** (rng.uniform(-8, 9, k) if i % 2 else rng.uniform(-1, 2, k))
        shells.append(dict(l=0, centre=c, expo=expo, coef=rng.uniform(0.1, 1.0, k)))
    sb = ShellBasis.from_shell_dicts(shells)
    ds = engine.DeviceShells(sb, "cuda")
    pairs = np.stack(np.tril_indices(sb.nshell), 1)
    ps = engine.PairSet(ds, pairs, max_exp=max_exp)
    if count:        # one warp a pair instead of several
        ps.ngroups = 0
        ps.build()
    rec = np.frombuffer(ps.p64.cpu().numpy().tobytes(), dtype="<f8").reshape(-1, 10)
    rec32 = np.frombuffer(ps.p32.cpu().numpy().tobytes(), dtype="<f4").reshape(-1, 12)
    kept = ps.kept.cpu().numpy()
    start = ps.prim_start.cpu().numpy()
    expo, coef, off = (x.cpu().numpy() for x in (ds.expo, ds.coef, ds.prim_off))
    q, eps = np.longdouble, 2.0 ** -53
    for n, (sa, s_b) in enumerate(pairs):
        AB = sb.centre[sa] - sb.centre[s_b]
        a, b = (x.ravel() for x in np.meshgrid(expo[off[sa]:off[sa + 1]], expo[off[s_b]:off[s_b + 1]],
                                               indexing="ij"))
        ca, cb = (x.ravel() for x in np.meshgrid(coef[off[sa]:off[sa + 1]],
                                                 coef[off[s_b]:off[s_b + 1]], indexing="ij"))
        ratio = a * b * float(AB @ AB) / (a + b)
        keep = ratio <= max_exp if max_exp > 0 else np.ones(len(a), bool)
        assert not np.any((np.abs(ratio - max_exp) < 1e-9 * max_exp) & (max_exp > 0))
        assert kept[n] == keep.sum()
        r = rec[start[n]:start[n] + kept[n]]
        a, b, ca, cb = (x[keep] for x in (a, b, ca, cb))
        assert np.array_equal(r[:, 0], a + b)
        ip = 1 / (q(1) * a + b)
        assert np.all(np.abs(r[:, 1] - ip / 2) <= 2 * eps * ip / 2 + eps * ip / 2)
        PA = -(b * ip)[:, None] * AB[None].astype(q)
        exact = sb.centre[sa].astype(q) - sb.centre[s_b].astype(q)     # AB before its rounding
        P = sb.centre[sa].astype(q)[None] - (b * ip)[:, None] * exact[None]
        # from the nearer centre: its step is at most half of AB
        step = np.minimum(a, b)[:, None] * ip[:, None] * np.abs(AB)[None]
        assert np.all(np.abs(r[:, 5:8] - PA) <= 5 * eps * np.abs(PA))
        assert np.all(np.abs(r[:, 2:5] - P) <= 5 * eps * step + eps * np.abs(P))
        x = a * (b * ip) * (AB.astype(q) @ AB.astype(q))
        K = q("5.914967172795612987") * ca * cb * ip * np.exp(-x)
        tiny = np.finfo(float).tiny
        assert np.all(np.abs(r[:, 8] - K) <= (10 + 10 * x) * eps * K + tiny)
        with np.errstate(under="ignore", over="ignore"):
            f = rec32[start[n]:start[n] + kept[n]]
            assert np.array_equal(f[:, :9], r[:, :9].astype(np.float32))
