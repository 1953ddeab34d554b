"""stats.bytes, the algorithmic bytes of a solve, against the arrays that the launches
read and write: V-cycles with and without levels in tiles, flexible CG, and flexible
GMRES between the passes that it needs and those that it may take."""
import pytest

from fortrancfd_gb300 import PressurePoisson
from tests import cases

pytestmark = pytest.mark.gpu


def _solve(c, tol=1e-7, **kw):
    """(bytes of the call, cycles, level sizes)"""
    with PressurePoisson(c.shape, c.spacing, **kw) as s:
        s.ppe_init(c.rho)
        _, st = s.solve(c.b, tol=tol)
        return st["bytes"], st["cycles"], [z * y * x for z, y, x in s.level_dims()]


def _level(n, nc):  # FP64, separate launches without a stored diagonal
    return 8.0 * (4 * 7 * n + 5 * n + 2 * nc + 2 * n + nc)


def test_vcycle_in_tiles(cuda):
    c = cases.config(0)  # 128 x 128: three levels in tiles, 16 x 16 in the block
    got, cyc, n = _solve(c)
    assert n == [16384, 4096, 1024, 256, 64]
    # two launches a level: p r/w, b, cx, cy, 1/diagonal; coarse b and e once each
    cycle = sum(8.0 * ((12 if l == 0 else 11) * n[l] + 2 * n[l + 1]) for l in range(3))
    cycle += _level(n[3], n[4]) + 8.0 * (2 * 64 + 64 * 64)
    rest = 40.0 * (cyc + 1) + 32.0 + 16.0   # residuals, mean, copies
    assert got == pytest.approx(cycle * cyc + rest * n[0], rel=1e-12)


def _vcycle(c):
    got, cyc, n = _solve(c)
    return (got - (40.0 * (cyc + 1) + 48.0) * n[0]) / cyc


def test_flexible_cg(cuda):
    c = cases.config(2, 16)  # 32^3: b - A p in every iteration
    got, cyc, n = _solve(c, krylov="fcg")
    # sum, dots, direction, A d, p, b - A p; the first residual, mean, copies
    want = _vcycle(c) * cyc + ((8 + 32 + 24 + 48 + 24 + 48) * cyc + 48 + 48) * n[0]
    assert got == pytest.approx(want, rel=1e-12)


def test_flexible_gmres(cuda):
    c = cases.config(2, 16)
    got, cyc, n = _solve(c, krylov="fgmres")
    assert 3 < cyc <= 30
    fixed = 24 + 8 * cyc + 16 + 48 + 48 + 48   # v_0, p += Z y, b - A p twice, mean, copies
    step = 8 + 16 + 48 + 24                    # sum, z_j, A z_j, v_{j+1}
    one = sum(16 * (j + 1) + 24 for j in range(cyc))   # a Gram-Schmidt pass
    base = _vcycle(c) * cyc + (fixed + step * cyc) * n[0]
    assert base + one * n[0] <= got * (1 + 1e-12)
    assert got <= (base + 2 * one * n[0]) * (1 + 1e-12)
