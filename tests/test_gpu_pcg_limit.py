"""Flexible CG at its cycle limit: b - A p decides, also where the recursion's
residual ends just above a tolerance that b - A p meets."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from tests import cases

pytestmark = pytest.mark.gpu


# (the last two are large enough for the recursion)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("index,scale", [(0, 2), (2, 16), (3, 1), (2, 4)])
def test_the_true_residual_decides_at_the_limit(cuda, precision, index, scale):
    c = cases.config(index, scale)
    for k in range(3, 10):
        with PressurePoisson(c.shape, c.spacing, precision=precision, krylov="fcg",
                             max_cycles=k) as s:
            s.ppe_init(c.rho)
            _, first = s.solve(c.b, tol=2e-11, check=False)  # all k cycles
            assert first["cycles"] == k and first["status"] == 1
            # the next larger tolerance, down to which the recursion has to go
            tol = float(np.nextafter(first["rel_residual"], 1.0))
            _, st = s.solve(c.b, tol=tol, check=False)
        assert st["rel_residual"] < tol and st["status"] == 0, k


# rows of one pair, two long rows, a box; coefficients from the density
# (colour-split FP32 level) and given (natural layout)
@pytest.mark.parametrize("form", ["rho", "coef"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape", [(1, 262144, 2), (1, 2, 262144), (64, 96, 64)])
def test_recursion_on_large_grids(cuda, shape, precision, form):
    """The same solution with the recursion (1e-9) and without (9e-12)."""
    nz, ny, nx = shape
    ext = (1.0, ny / nx, nz / nx if nz > 1 else 1.0)
    c = cases.Built(inputs.custom(shape, extent=ext, radii=(0.3,), seed=3,
                                  centers=((0.5, 0.4 * ext[1], 0.5 * ext[2]),)))
    with PressurePoisson(c.shape, c.spacing, precision=precision, krylov="fcg",
                         max_cycles=100) as s:
        if form == "rho":
            s.ppe_init(c.rho)
        else:
            s.set_coef(*c.coef)
        p, st = s.solve(c.b, tol=1e-9)
        q, st2 = s.solve(c.b, tol=9e-12)
    assert st["rel_residual"] < 1e-9 and st2["rel_residual"] < 9e-12
    # two residuals of 1e-9 |b| apart, and the smoothest mode's eigenvalue
    bound = 1e-9 * np.linalg.norm(c.b) * 1000.0 * (max(ext) / np.pi) ** 2
    assert np.linalg.norm(p - q) <= bound
