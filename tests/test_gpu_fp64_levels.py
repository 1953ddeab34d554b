"""The FP64 cycle's half restriction (the colour relaxed last has no residual),
its one-colour prolongation and its one-block bottom: the iterate after each
cycle against the oracle's full restriction, over grids with one-cell axes, odd
coarse levels, one sweep or none before and after the coarse correction, and a
bottom of every size around the one-block limit."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from oracle import oracle as orc
from tests import cases
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu


# finest first: 2D, an axis of one cell in x, odd coarsest axes, 1024 cells on
# level 1 (in one block) and 1536 (separate launches), two levels only
@pytest.mark.parametrize("shape", [(1, 64, 64), (16, 32, 1), (12, 20, 12), (1, 96, 64),
                                   (16, 16, 32), (1, 8, 16)])
@pytest.mark.parametrize("nu", [(2, 2), (1, 0), (0, 1), (3, 1)])
def test_iterates_match_oracle(cuda, shape, nu):
    nz, ny, nx = shape
    n = max(shape)
    ext = tuple(m / n if m > 1 else 1.0 for m in (nx, ny, nz))
    c = cases.Built(inputs.custom(shape, extent=ext, radii=(0.2,), seed=3,
                                  centers=(tuple(0.45 * e for e in ext),)))
    for k in (1, 2):
        want, _ = orc.mg_solve(c.coef, c.b, tol=1e-300, max_cycles=k, nu1=nu[0], nu2=nu[1])
        with PressurePoisson(c.shape, c.spacing, max_cycles=k, nu1=nu[0], nu2=nu[1]) as s:
            s.ppe_init(c.rho)
            p, st = s.solve(c.b, tol=1e-300, check=False)
        assert st["cycles"] == k
        # as the per-cycle parity test: rounding only
        assert rel_l2(p - p.mean(), want - want.mean()) <= 1e-12, k
