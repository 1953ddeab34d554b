"""Flexible CG at its cycle limit: b - A p decides, also where the recursion's
residual ends just above a tolerance that b - A p meets."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("index,scale", [(0, 2), (2, 16)])
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
