"""The FP32 Boys function in float pairs: as exact as FP64 values rounded once."""
import numpy as np
import pytest

import hostcheck

ASYM32 = [17, 20, 23, 25, 28, 30, 32, 34, 36, 38]


def boys(m, t):
    """F_0..F_m(t) in long double: the series of F_m, all terms positive, and downward recursion."""
    t = t.astype(np.longdouble)
    e = np.exp(-t)
    term = np.full_like(t, np.longdouble(1) / (2 * m + 1))
    total = term.copy()
    for i in range(1, 300):
        term = term * (2 * t / (2 * m + 2 * i + 1))
        total += term
    f = [e * total]
    for k in range(m, 0, -1):
        f.insert(0, (2 * t * f[0] + e) / (2 * k - 1))
    return np.stack(f, 1)


@pytest.mark.parametrize("m", range(10))
def test_boys_pair32_rounds_once(m):
    """Half a unit in the last place (at least 2^-24 of the value) of the one rounding, the terms left
    out, (1/32)^5 / 5! = 2^-31.9 of the value or 0.005 units, and the expansions' roundings at
    2^-35, below 0.003: 0.51 units.  The rms is that of rounding exact values to 1e-3 of it."""
    L = hostcheck.hc()
    rng = np.random.default_rng(100 + m)
    t = np.concatenate([rng.uniform(0.0, ASYM32[m], 2000),
                        np.exp(rng.uniform(np.log(1e-4), np.log(ASYM32[m]), 2000))])
    t = t.astype(np.float32).astype(float)
    t = t[t < ASYM32[m]]
    exact = boys(m, t)
    got = np.zeros((len(t), m + 1))
    for x, row in zip(t, got):
        assert L.hc_boys_pair32(m, float(x), row.ctypes.data) == 0
    unit = np.spacing(exact.astype(np.float32)).astype(float)
    rms = lambda y: float(np.sqrt(np.mean(((y - exact) / unit).astype(float) ** 2)))   # noqa: E731
    assert np.max(np.abs(got - exact) / unit) <= 0.51
    assert rms(got) <= 1.001 * rms(exact.astype(np.float32).astype(float))
