"""Without pre-smoothing the finest FP32 unknown is set to zero before a cycle, all of it:
a solve after one that went to NaN is a fresh handle's solve, bit for bit."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("krylov", ["none", "fcg", "fgmres"])
@pytest.mark.parametrize("index,scale", [(0, 1), (1, 8)])
def test_solve_after_a_failed_one(cuda, index, scale, krylov):
    c = cases.config(index, scale)
    kw = dict(precision="mixed", krylov=krylov, nu1=0, max_cycles=40)
    out = []
    for fail in (False, True):
        with PressurePoisson(c.shape, c.spacing, **kw) as s:
            s.ppe_init(c.rho)
            if fail:
                s.solve(np.full_like(c.b, np.nan), tol=1e-8, check=False)
            out.append(s.solve(c.b, tol=1e-8, check=False)[0])
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])
