"""The cells outside the interface band are left out of redistancing's sums only where
they add nothing: with a density ratio near the largest double the weight's other
factor overflows, times delta = 0 it is a NaN, and the NaN spreads as in the oracle."""
import numpy as np
import pytest

from fortrancfd_gb300 import LevelSet
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

RATIOS = [1e-3, 1e70, 1.5e308]


def _phi(shape):
    z, y, x = np.meshgrid(*[np.arange(n) + 0.5 for n in shape], indexing="ij")
    r = np.sqrt((x - 0.4 * shape[2]) ** 2 + (y - 0.5 * shape[1]) ** 2 + (z - 0.5 * shape[0]) ** 2)
    return (r - 0.3 * max(shape)) / max(shape)


@pytest.mark.parametrize("rho_12", RATIOS)
def test_redistance(cuda, rho_12):
    shape, h = (10, 20, 24), 1.0 / 24
    phi = _phi(shape)
    with np.errstate(all="ignore"):
        want, it_w, _ = orc.ls_redistance(phi, 1.5 * h, 0.1 * h, (h, h, h), rho_12=rho_12, btn=1,
                                          max_iter=3)
    got = phi.copy()
    with LevelSet(shape, (h, h, h)) as ls:
        _, it, _ = ls.redistance(got, 1.5 * h, 0.1 * h, rho_12, btn=1, max_iter=3)
    assert it == it_w
    # sin and cos of two libraries
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(phi).max())
