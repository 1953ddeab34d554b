"""The bottom of the FP32 cycle in one block against the same levels as separate
launches: the same arithmetic in the same order, so the iterates are the same
bits.  One-cell axes, a coarsened z alone (its slopes start where no x or y slopes
lie), an odd coarsest width, levels that are no powers of two, more than two pairs
per thread, and each count of sweeps down to none."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, inputs
from tests import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(256, 1, 1), (1, 1, 512), (1, 256, 1), (32, 16, 16),
                                   (16, 24, 40), (32, 24, 1), (8, 1, 64), (1, 72, 56),
                                   (128, 128, 1)])
@pytest.mark.parametrize("nu", [(2, 2), (1, 0), (0, 1), (3, 1)])
def test_same_bits_as_separate_launches(cuda, monkeypatch, shape, nu):
    nz, ny, nx = shape
    n = max(shape)
    ext = tuple(m / n if m > 1 else 1.0 for m in (nx, ny, nz))
    c = cases.Built(inputs.custom(shape, extent=ext, radii=(0.2,), seed=3,
                                  centers=(tuple(0.45 * e for e in ext),)))
    got = []
    for flag in ("0", "1"):
        monkeypatch.setenv("GBMG_SUBCYCLE", flag)
        with PressurePoisson(c.shape, c.spacing, max_cycles=3, nu1=nu[0], nu2=nu[1],
                             precision="mixed") as s:
            s.ppe_init(c.rho)
            p, st = s.solve(c.b, tol=1e-300, check=False)
        got.append(p)
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_a_smaller_handle_leaves_an_earlier_one_alone(cuda, precision):
    """The block's shared-memory limit is the kernel's, shared by all handles."""
    big, small = cases.config(1, 8), cases.Built(inputs.custom(
        (1, 16, 16), extent=(1.0, 1.0, 1.0), radii=(0.2,), seed=3, centers=((0.5, 0.5, 0.5),)))
    with PressurePoisson(big.shape, big.spacing, precision=precision) as s:
        with PressurePoisson(small.shape, small.spacing, precision=precision) as t:
            t.ppe_init(small.rho)
            t.solve(small.b, tol=1e-8)
            s.ppe_init(big.rho)
            _, st = s.solve(big.b, tol=1e-8)
    assert st["status"] == 0
