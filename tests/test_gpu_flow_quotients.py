"""The projection's quotients (face coefficients, divergence, correction,
divergence statistics) on spacings that are and are not powers of two: bit for
bit the oracle's or numpy's divisions."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,spacing", [((1, 24, 40), (0.03, 0.25, 1.0)),
                                           ((8, 12, 20), (1.0 / 48, 0.017, 1.0 / 3)),
                                           ((16, 16, 16), (1.0 / 16, 1.0 / 16, 1.0 / 16))])
def test_bitwise(cuda, shape, spacing):
    rng = np.random.default_rng(5)
    nz, ny, nx = shape
    rho = np.where(rng.random(shape) < 0.4, 1.0, 1000.0 * rng.random(shape) + 0.1)
    u, v, w = (rng.standard_normal(s) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx),
                                                (nz + 1, ny, nx)))
    if nz == 1:
        w[...] = 0.0
    u[..., 3:6] = 0.25
    v[:, 2:5] = -0.0
    dt = 0.007
    with PressurePoisson(shape, spacing, krylov=True, max_cycles=300) as s:
        s.ppe_init(rho)
        for a, b in zip(s.level_coef(0), orc.face_coef(rho, spacing)):
            np.testing.assert_array_equal(a, b)
        wd = w if nz > 1 else None
        # (the oracle's divergence has its mean removed)
        div = (u[..., 1:] - u[..., :-1]) / spacing[0] + (v[:, 1:] - v[:, :-1]) / spacing[1]
        if nz > 1:
            div = div + (w[1:] - w[:-1]) / spacing[2]
        np.testing.assert_array_equal(s.divergence(u, v, wd, dt), div / dt)
        mx, mean = s.div_stats(u, v, wd)
        d = np.abs(div)
        assert mx == d.max() and abs(mean - d.mean()) <= 1e-14 * d.mean()
        uc, vc, wc = u.copy(), v.copy(), w.copy()
        p, _ = s.ppe_solver(uc, vc, wc if nz > 1 else None, dt, tol=1e-8, check=False)
        want = orc.correct(rho, p, dt, u, v, w, spacing)
        for a, b in zip((uc, vc, wc)[: 3 if nz > 1 else 2], want):
            np.testing.assert_array_equal(a, b)
