"""The kernels' own elementary functions against extended precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def ulps(y, exact):
    """Errors of the doubles y in units in the last place of the long doubles ``exact``."""
    return np.abs((y.astype(np.longdouble) - exact) / np.spacing(exact.astype(float))).astype(float)


def test_rsqrt_is_as_exact_as_the_library(gpu_lib):
    """Half a unit of the last rounding, the step's own error, 5/16 r^3 with |r| <= 2^-19 (2^-58.6 of
    the value, 0.02 units at most), and the roundings of the correction, 2^-19 of half a unit each:
    0.53 at most.  The rms is a rounding's, 1/sqrt(12), to 1 %."""
    from gaussium_gb300 import _lib
    rng = np.random.default_rng(8)
    x = np.concatenate([rng.uniform(1.0, 4.0, 400000),
                        np.exp(rng.uniform(np.log(2.3e-308), np.log(1.7e308), 400000)),
                        [2.2250738585072014e-308, 1.7976931348623157e308]])
    d = torch.as_tensor(x).cuda()
    y = torch.empty_like(d)
    _lib.check(gpu_lib.gs_rsqrt_eval(len(x), _lib.ptr(d), _lib.ptr(y), _lib.stream()), "rsqrt")
    e = ulps(y.cpu().numpy(), 1 / np.sqrt(x.astype(np.longdouble)))
    assert e.max() <= 0.53 and np.sqrt((e * e).mean()) <= 1.01 / np.sqrt(12.0)
