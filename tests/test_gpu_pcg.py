"""The flexible-CG passes (pcg.cu): the pair mapping of the colour-split and
natural layouts on small and odd grids, the residual recursion against the
residual recomputed every iteration (tolerances under 1e-11), and a handle that
changes between the two."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from oracle import oracle as orc
from tests import cases
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu


def _built(shape):
    nz, ny, nx = shape
    ext = (1.0, ny / nx, nz / nx if nz > 1 else 1.0)
    return cases.Built(inputs.custom(shape, extent=ext, radii=(0.3 * min(ext[:2]),), seed=3,
                                     centers=((0.5, 0.4 * ext[1], 0.5 * ext[2]),)))


# odd cells without a coarser level, rows of one pair, three pairs, a plane of
# one row pair, several rows per block
@pytest.mark.parametrize("shape", [(1, 7, 9), (3, 3, 5), (1, 64, 2), (2, 2, 2), (1, 12, 6),
                                   (4, 6, 10), (16, 24, 40)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_matches_oracle_on_small_grids(cuda, shape, precision):
    c = _built(shape)
    want, _ = orc.mg_solve(c.coef, c.b, tol=1e-13, max_cycles=400, krylov=1)
    with PressurePoisson(c.shape, c.spacing, precision=precision, krylov="fcg",
                         max_cycles=200) as s:
        s.ppe_init(c.rho)
        p, st = s.solve(c.b, tol=1e-10)
    assert st["status"] == 0 and st["rel_residual"] < 1e-10
    assert rel_l2(p, want) <= 1e-9  # the whole-solve bound of the parity tests


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_recursion_and_recomputed_residual(cuda, precision):
    """The reported residual is b - A p whichever way the loop got it, and a
    handle that alternates between the two gives a fresh handle's bits."""
    c = cases.config(2, 8)
    kw = dict(precision=precision, krylov="fcg", max_cycles=300)
    alone = {}
    for tol in (1e-10, 1e-12):
        with PressurePoisson(c.shape, c.spacing, **kw) as s:
            s.ppe_init(c.rho)
            alone[tol] = s.solve(c.b, tol=tol)[0]
    with PressurePoisson(c.shape, c.spacing, **kw) as s:
        s.ppe_init(c.rho)
        for tol in (1e-10, 1e-12, 1e-10, 1e-12):
            p, st = s.solve(c.b, tol=tol)
            assert st["status"] == 0 and st["rel_residual"] < tol
            np.testing.assert_array_equal(p, alone[tol])
            b = c.b - c.b.mean()
            _, n2 = s.residual(b, p, want_r=False)
            # the mean projection after the loop moves p by rounding only
            assert abs(np.sqrt(n2) / np.linalg.norm(b) - st["rel_residual"]) <= 1e-13
    assert rel_l2(alone[1e-10], alone[1e-12]) <= 1e-9
