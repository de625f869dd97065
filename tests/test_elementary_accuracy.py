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


def evaluate(gpu_lib, name, x):
    from gaussium_gb300 import _lib
    d = torch.as_tensor(np.asarray(x, dtype=np.float64)).cuda()
    y = torch.empty_like(d)
    _lib.check(getattr(gpu_lib, name)(len(d), _lib.ptr(d), _lib.ptr(y), _lib.stream()), name)
    return y.cpu().numpy()


def test_rcp(gpu_lib):
    """Half a unit of the last rounding and the series' rest, e^3 with |e| <= 2^-19.9: 0.51 units.
    Outside its range the division's own values."""
    rng = np.random.default_rng(9)
    x = np.concatenate([rng.uniform(1.0, 2.0, 400000),
                        np.exp(rng.uniform(np.log(2.3e-308), np.log(4.4e307), 400000)),
                        [2.2250738585072014e-308, 2.0 ** 1021, np.nextafter(2.0 ** 1022, 0)]])
    assert ulps(evaluate(gpu_lib, "gs_rcp_eval", x), 1 / x.astype(np.longdouble)).max() <= 0.51
    odd = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0 ** 1022, 2.0 ** 1023, 1.7e308, np.inf, -np.inf,
                    np.nan, -3.0, -1e-310])
    with np.errstate(divide="ignore", over="ignore"):
        assert np.array_equal(evaluate(gpu_lib, "gs_rcp_eval", odd), 1.0 / odd, equal_nan=True)


def test_exp(gpu_lib):
    """In units of 2^-53 of a value from 0.7 to 1.42 (times a power of two): the last rounding half a
    unit in the last place, the reduced argument's 0.25, the sum's roundings 0.35 and 0.06, the float
    terms' 0.11, the terms left out 0.03: 1.3 units in the last place.  From |x| = 700 on the
    library's own values."""
    rng = np.random.default_rng(10)
    x = np.concatenate([rng.uniform(-700, 700, 400000), rng.uniform(-2, 2, 400000),
                        -np.exp(rng.uniform(np.log(1e-18), 0, 1000)), [0.0, -0.0, 699.9999, -699.9999]])
    e = ulps(evaluate(gpu_lib, "gs_exp_eval", x), np.exp(x.astype(np.longdouble)))
    assert e.max() <= 1.3
    odd = np.array([700.0, -700.0, 709.7, 710.0, -708.0, -740.0, -746.0, np.inf, -np.inf, np.nan])
    lib = torch.exp(torch.as_tensor(odd).cuda()).cpu().numpy()
    assert np.array_equal(evaluate(gpu_lib, "gs_exp_eval", odd), lib, equal_nan=True)
