"""Flexible GMRES's vector passes (products in groups of one to eight basis vectors,
the update with the norm, the scaled vector written in the V-cycle's layout) over
odd and even cell counts, FP64 and FP32 levels in both layouts, a preconditioner
from a zero guess with no sweeps before the coarse correction, and enough steps for
every group size: the true FP64 residual and the oracle's solution, as the
parity test of the same solver asks."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from oracle import oracle as orc
from tests import cases
from tests.cases import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 7, 7), (1, 24, 40), (16, 24, 40), (1, 128, 64)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nu", [(2, 2), (1, 0), (0, 1)])
def test_residual_and_solution(cuda, shape, precision, nu):
    nz, ny, nx = shape
    n = max(shape)
    ext = tuple(m / n if m > 1 else 1.0 for m in (nx, ny, nz))
    c = cases.Built(inputs.custom(shape, extent=ext, radii=(0.2,), seed=3,
                                  centers=(tuple(0.45 * e for e in ext),)))
    want, st_or = orc.mg_solve(c.coef, c.b, tol=1e-10, krylov=1)
    assert st_or["status"] == 0
    out = []
    for graph in (True, False):
        with PressurePoisson(c.shape, c.spacing, precision=precision, krylov="fgmres",
                             max_cycles=400, nu1=nu[0], nu2=nu[1], use_graph=graph) as s:
            s.ppe_init(c.rho)
            p, st = s.solve(c.b, tol=1e-10)
        assert st["status"] == 0
        out.append(p)
    _, r2 = orc.residual(c.coef, p, c.b)
    assert np.sqrt(r2) / np.linalg.norm(c.b) < 1e-10
    assert rel_l2(p, want) <= 1e-9
    assert np.array_equal(out[0], out[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cycle_limit_and_restart(cuda, precision):
    """The V-cycle launched ahead of the host's tests ends with the cycle limit and
    with the basis (30 vectors): the asked number of steps, the reported residual
    that of the returned p in FP64 (its norms differ by rounding, 1e-10 of it here:
    it stays above 1e-5 of b), never larger after more steps."""
    shape = (1, 128, 64)
    c = cases.Built(inputs.custom(shape, extent=(0.5, 1.0, 1.0), radii=(0.2,), seed=3,
                                  centers=((0.25, 0.5, 0.5),)))
    rels = []
    for k in (1, 2, 5, 29, 30, 31, 61):
        # (one sweep before the coarse correction alone: many steps)
        with PressurePoisson(c.shape, c.spacing, precision=precision, krylov="fgmres",
                             max_cycles=k, nu1=1, nu2=0) as s:
            s.ppe_init(c.rho)
            p, st = s.solve(c.b, tol=1e-300, check=False)
        _, r2 = orc.residual(c.coef, p, c.b)
        rel = np.sqrt(r2) / np.linalg.norm(c.b)
        assert st["cycles"] == k
        if rel > 1e-5:
            assert abs(st["rel_residual"] - rel) <= 1e-10 * rel
            rels.append(rel)
    assert len(rels) >= 2
    assert all(b <= a * (1 + 1e-6) for a, b in zip(rels, rels[1:]))
