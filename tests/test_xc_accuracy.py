"""Rounding of the exchange-correlation matrix's sums over the grid."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npts,n", [(64800, 8), (129599, 5)])
def test_matrix_rounding(gpu_lib, npts, n):
    """Elements that are sums of npts terms of one sign, against long double.  With u = 2^-53 and
    0.58 u the rms rounding of one addition: about 300 parts of some 200 to 450 points (their own
    chains' errors, 0.58 u sqrt(450 / 3), average over the parts to 0.4 u), added in eight chains
    of 38 (0.58 u sqrt(38 / 3) / sqrt(8) = 0.7 u) and a tree of three levels (1.0 u): 1.3 u rms in
    all.  Twice that is allowed; one chain over the parts has 0.58 u sqrt(304 / 3) = 5.8 u."""
    from gaussium_gb300 import _lib
    rng = np.random.default_rng(npts)
    phi = rng.uniform(0.1, 1.0, (npts, n))
    p = np.eye(n) + 0.1
    w = rng.uniform(0.1, 1.0, npts)
    up = lambda a: torch.as_tensor(a).cuda()      # noqa: E731
    need = gpu_lib.gs_xc_lda_workspace(npts, n)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    v = torch.empty((n, n), dtype=torch.float64, device="cuda")
    e = torch.empty((), dtype=torch.float64, device="cuda")
    phi_d, p_d, w_d = up(phi), up(p), up(w)
    alpha = 2 / 3
    _lib.check(gpu_lib.gs_xc_lda(npts, n, _lib.ptr(phi_d), _lib.ptr(p_d), _lib.ptr(w_d), alpha, 0,
                                 0.0, 0.0, 0.0, 1.0, _lib.ptr(v), _lib.ptr(e), _lib.ptr(ws), need,
                                 _lib.stream()), "gs_xc_lda")
    ld = np.longdouble
    ph = phi.astype(ld)
    rho = ((ph @ p.astype(ld)) * ph).sum(1)
    # the weighted potential of the rounded density, from the library: its constants' roundings are
    # the same at every point and no part of the sums
    r, wv, we = up(rho.astype(float)), torch.empty_like(w_d), torch.empty_like(w_d)
    _lib.check(gpu_lib.gs_lda_xc(npts, _lib.ptr(r), _lib.ptr(w_d), alpha, 0, 0.0, 0.0, 0.0, 1.0,
                                 _lib.ptr(wv), _lib.ptr(we), _lib.stream()), "gs_lda_xc")
    ref = ph.T @ (ph * wv.cpu().numpy().astype(ld)[:, None])
    err = np.abs((v.cpu().numpy() - ref) / ref).astype(float)
    assert np.sqrt((err ** 2).mean()) <= 2.6 * 2.0 ** -53
