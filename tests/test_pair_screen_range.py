"""The primitive-pair screen's float test where its products leave float's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_screen_of_huge_exponents(gpu_lib):
    """Pairs of exponents up to 1e30 on centres so close that ab/p |AB|^2 is far below the limit, or
    far above it: kept or dropped as in double, by both kernels."""
    from gaussium_gb300 import engine
    from gaussium_gb300.basis import ShellBasis
    shells = [dict(l=0, centre=np.zeros(3), expo=np.array([a]), coef=np.ones(1))
              for a in (1e20, 1e30, 1.0)]
    shells += [dict(l=0, centre=np.array([d, 0.0, 0.0]), expo=np.array([a]), coef=np.ones(1))
               for d in (1e-12, 1e-16, 1e-3, 1e20) for a in (1e20, 1e30, 3e-9)]
    sb = ShellBasis.from_shell_dicts(shells)
    pairs = np.stack(np.tril_indices(sb.nshell), 1)
    ps = engine.PairSet(engine.DeviceShells(sb), pairs, max_exp=55.0)
    a, b = sb.expo[pairs[:, 0]], sb.expo[pairs[:, 1]]
    ab2 = ((sb.centre[pairs[:, 0]] - sb.centre[pairs[:, 1]]) ** 2).sum(1)
    x = a * b * ab2 / (a + b)
    assert not np.any(np.abs(x - 55.0) < 1e-6 * 55.0)
    for form in range(2):
        if form:                       # one warp a pair instead of several
            ps.ngroups = 0
            ps.build()
        assert np.array_equal(ps.kept.cpu().numpy()[:ps.n], x <= 55.0)
    assert np.any(x > 55.0) and np.any((x < 1.0) & (a * b > 1e39) & (ab2 > 0.0))
