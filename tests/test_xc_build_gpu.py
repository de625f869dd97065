"""``gs_xc_lda``, one exchange-correlation build, against the same contractions with torch."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 100), (3, 31), (4, 32), (5, 33), (8, 64), (9, 65), (16, 1), (17, 700),
         (33, 12345), (76, 4099), (129, 2000), (263, 1000), (440, 333)]


def build(gpu_lib, phi, p, w, alpha, vwn):
    from gaussium_gb300 import _lib
    npts, n = phi.shape
    need = gpu_lib.gs_xc_lda_workspace(npts, n)
    ws = torch.full((need,), 255, dtype=torch.uint8, device="cuda")
    v = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    e = torch.full((), float("nan"), dtype=torch.float64, device="cuda")
    a, x0, b, c = vwn if vwn is not None else (0.0, 0.0, 0.0, 1.0)
    _lib.check(gpu_lib.gs_xc_lda(npts, n, _lib.ptr(phi), _lib.ptr(p), _lib.ptr(w), alpha,
                                 int(vwn is not None), a, x0, b, c, _lib.ptr(v), _lib.ptr(e),
                                 _lib.ptr(ws), need, _lib.stream()), "gs_xc_lda")
    return v, e


@pytest.mark.parametrize("n,npts", SIZES)
def test_matches_torch(gpu_lib, n, npts):
    """Sums of up to N^2 and npts terms in another order, and functionals of densities that
    differ in their last bits (a few parts in 1e12 through the correlation's cancelling
    logarithms): 1e-11 of the sums of magnitudes.  The density is not symmetric: only its
    symmetric part enters."""
    rng = np.random.default_rng(n + npts)
    phi = torch.as_tensor(rng.standard_normal((npts, n))).cuda()
    c = rng.standard_normal((n, max(1, n // 3)))
    k = rng.standard_normal((n, n))
    p = torch.as_tensor(c @ c.T + k - k.T).cuda()
    w = torch.as_tensor(rng.uniform(0.1, 1.0, npts)).cuda()
    v, e = build(gpu_lib, phi, p, w, 2 / 3, oracle.VWN3)
    rho = ((phi @ p) * phi).sum(1).cpu().numpy()
    e_ref, v_ref = oracle._xc_parts(np.where(rho > 1e-300, rho, 0.0), 2 / 3, oracle.VWN3)
    ok = rho > 1e-300
    wv = w * torch.as_tensor(np.where(ok, v_ref, 0.0)).cuda()
    ref = phi.T @ (phi * wv[:, None])
    scale = phi.abs().T @ (phi.abs() * wv.abs()[:, None])
    assert float(((v - ref).abs() - 1e-11 * scale).max()) <= 0.0
    assert torch.equal(v, v.T)
    we = w.cpu().numpy() * np.where(ok, rho * e_ref, 0.0)
    assert abs(float(e) - we.sum()) <= 1e-11 * np.abs(we).sum()
    v2, e2 = build(gpu_lib, phi, p, w, 2 / 3, oracle.VWN3)
    assert torch.equal(v, v2) and float(e) == float(e2)


def test_refusals_and_fallback(gpu_lib):
    """Too many functions, a bad fit and a short workspace are refused; a density torch
    refuses stays refused."""
    from gaussium_gb300 import _lib
    from gaussium_gb300.kohnsham import ExchangeCorrelationGPU
    from molecules import load
    x = torch.ones(1 << 20, dtype=torch.float64, device="cuda")
    q = _lib.ptr(x)

    def call(n, vwn_c=42.0, ws=1 << 22):
        return gpu_lib.gs_xc_lda(8, n, q, q, q, 0.7, 1, 0.06, -0.1, 10.0, vwn_c, q, q, q, ws, None)
    assert call(gpu_lib.gs_xc_lda_max_functions() + 1) == 6
    assert call(4, vwn_c=1.0) == 1 and call(4, ws=64) == 5 and call(0) == 1
    xc = ExchangeCorrelationGPU(load("h2o_sto3g")[1], params=(2 / 3, None), radial=4)
    p = torch.eye(7, dtype=torch.float64, device="cuda")
    v, _ = xc.evaluate_device(p.t())
    assert torch.equal(v, xc.evaluate_device(p)[0])
    for bad in (p.float(), torch.eye(6, dtype=torch.float64, device="cuda"), p.cpu()):
        with pytest.raises(RuntimeError):
            xc.evaluate_device(bad)
