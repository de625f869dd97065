"""Which exchange-correlation builds go to ``gs_xc_lda`` and which through torch."""
import types

import pytest
import torch

from gaussium_gb300 import kohnsham


def refuse(rc, what):
    assert rc == 0, what


def builder(npts, n):
    """An ExchangeCorrelationGPU on the CPU whose functionals are v = 2 rho, eps = rho."""
    xc = object.__new__(kohnsham.ExchangeCorrelationGPU)
    g = torch.Generator().manual_seed(n)
    xc.sb, xc.device, xc.alpha, xc.vwn = types.SimpleNamespace(nbf=n), torch.device("cpu"), 0.7, None
    xc._phi = torch.randn((npts, n), dtype=torch.float64, generator=g)
    xc.weights = torch.rand(npts, dtype=torch.float64, generator=g)
    xc.functionals = lambda rho, w: (2.0 * w * rho, w * rho * rho)
    return xc


@pytest.mark.parametrize("kind", ["no points", "negated view", "sparse", "phi of other strides",
                                  "large", "plain"])
def test_route(kind, monkeypatch):
    calls = []

    class Library:
        def gs_xc_lda_max_functions(self):
            return 4

        def gs_xc_lda_workspace(self, npts, n):
            return 16

        def gs_xc_lda(self, npts, *a):
            calls.append(npts)
            return 0 if npts > 0 else 1              # as the library: no points is an error
    monkeypatch.setattr(kohnsham._lib, "lib", Library)
    monkeypatch.setattr(kohnsham._lib, "stream", lambda: None)
    monkeypatch.setattr(kohnsham._lib, "check", refuse)
    n = 5 if kind == "large" else 3
    xc = builder(0 if kind == "no points" else 11, n)
    a = torch.randn((n, n), dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    a = a + a.T
    p = a
    if kind == "negated view":
        p = torch.complex(a, -a).conj().imag         # holds -a behind a negative bit
        assert p.is_neg()
    elif kind == "sparse":
        p = a.to_sparse_csr()
    elif kind == "phi of other strides":
        xc._phi = xc._phi.T.contiguous().T
    phi = xc._phi
    v, e = xc.evaluate_device(p)
    assert calls == ([11] if kind == "plain" else [])
    if kind == "plain":
        return
    rho = ((phi @ a) * phi).sum(1)
    ref = phi.T @ (phi * (2.0 * xc.weights * rho)[:, None])
    assert v.shape == (n, n) and torch.allclose(v, ref, rtol=1e-12, atol=1e-12)
    assert torch.allclose(e, (xc.weights * rho * rho).sum())


@pytest.mark.gpu
def test_grid_without_points(gpu_lib):
    from molecules import load
    xc = kohnsham.ExchangeCorrelationGPU(load("h2o_sto3g")[1], params=(2 / 3, kohnsham.VWN3), radial=0)
    v, e = xc.evaluate_device(torch.eye(7, dtype=torch.float64, device="cuda"))
    assert v.shape == (7, 7) and not v.any() and float(e) == 0.0
