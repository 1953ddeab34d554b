"""2D levels of the cycle by tiles against the same levels as separate
launches: the same arithmetic in the same order, so the iterates are the same
bits.  Levels that end inside a tile, one and two sweeps per launch, sweep counts
whose launches add up to odd and even (the unknown changes its array with each),
a zero and a given start of the finest FP64 level, both orders of colours."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,precision", [
    ((1, 320, 192), "mixed"), ((1, 224, 288), "mixed"), ((1, 512, 640), "mixed"),
    ((1, 128, 48), "mixed"), ((1, 112, 144), "fp64"), ((1, 256, 96), "fp64"),
    ((1, 512, 512), "fp64"), ((1, 56, 24), "fp64")])
@pytest.mark.parametrize("nu,krylov", [((2, 2), "none"), ((1, 2), "none"), ((3, 2), "none"),
                                       ((2, 2), "fcg"), ((1, 1), "fcg")])
def test_same_bits_as_separate_launches(cuda, monkeypatch, shape, precision, nu, krylov):
    nz, ny, nx = shape
    n = max(shape)
    ext = tuple(m / n if m > 1 else 1.0 for m in (nx, ny, nz))
    c = cases.Built(inputs.custom(shape, extent=ext, radii=(0.2,), seed=3,
                                  centers=(tuple(0.45 * e for e in ext),)))
    got = []
    monkeypatch.setenv("GBMG_SUBCYCLE", "0")   # (the block's FP64 coarse sums have an order of their own)
    for flag in ("0", "1"):
        monkeypatch.setenv("GBMG_TILES", flag)
        with PressurePoisson(c.shape, c.spacing, max_cycles=3, nu1=nu[0], nu2=nu[1],
                             precision=precision, krylov=krylov) as s:
            s.ppe_init(c.rho)
            p, _ = s.solve(c.b, tol=1e-300, check=False)
        got.append(p)
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])
