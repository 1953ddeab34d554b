"""Flexible CG near the accuracy that FP64 allows, where the recursion's residual strays
from b - A p by as much as the tolerance.  Four bubbles of ratio 1000 on fine 2D
grids: just above 1e-11 a solve takes the cycles that it takes just below (b - A p
in every iteration), up to the one or two that rounding decides; steered by a
residual that far off it took ten more.  Four of ratio 1e5 in 3D: the solve
converges (in 22 to 27 cycles with b - A p in every iteration), where it stuck."""
import numpy as np
import pytest
import torch

from fortrancfd_gb300 import PressurePoisson, inputs

pytestmark = pytest.mark.gpu


AT = [(0.25, 0.3, 0.5), (0.25, 0.7, 0.5), (0.75, 0.3, 0.5), (0.75, 0.7, 0.5)]


def _rhs(shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    b = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    return b - b.mean()


@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [512, 1024])
def test_cycles_near_the_floor(cuda, n, precision, use_graph):
    case = inputs.custom((1, n, n), centers=AT, radii=(0.12,) * 4)
    phi = torch.from_numpy(inputs.level_set(case)).to(cuda)
    with PressurePoisson(case.shape, case.spacing, precision=precision, krylov="fcg",
                         max_cycles=100, use_graph=use_graph) as s:
        s.rho_mu(phi, case.eps, 1000.0, 1.0)
        for seed in range(6):
            b = _rhs(case.shape, seed)
            above, below = (s.solve(b, tol=t)[1] for t in (1.1e-11, 0.99e-11))
            assert above["rel_residual"] < 1.1e-11
            assert above["cycles"] <= below["cycles"] + 2, seed
            # a start close to the solution goes without the recursion
            p = s.solve(b, tol=1e-9)[0]
            _, warm = s.solve(b, p, tol=1.1e-11)
            assert warm["rel_residual"] < 1.1e-11
            assert np.isfinite(p.cpu().numpy()).all()


@pytest.mark.parametrize("use_graph", [True, "cycle", False])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [64, 256])
def test_large_density_ratio(cuda, n, precision, use_graph):
    case = inputs.custom((n, n, n), centers=AT, radii=(0.12,) * 4)
    phi = torch.from_numpy(inputs.level_set(case)).to(cuda)
    with PressurePoisson(case.shape, case.spacing, precision=precision, krylov="fcg",
                         max_cycles=32, use_graph=use_graph) as s:
        s.rho_mu(phi, case.eps, 1e5, 1.0)
        for seed in range(2 if n == 256 else 6):
            for tol in (1e-9, 1e-10, 3e-11):
                st = s.solve(_rhs(case.shape, seed), tol=tol, check=False)[1]
                assert st["status"] == 0 and st["rel_residual"] < tol, (seed, tol)
