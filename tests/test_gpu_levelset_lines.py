"""The line segments of the level-set kernels (64 cells, 59 faces complete per
segment, eight lines per block) at their edges, and the split fluxes that are
zero on a stencil: bit for bit the oracle."""
import numpy as np
import pytest

from fortrancfd_gb300 import LevelSet
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [(1, 7, 58), (1, 59, 9), (2, 60, 61), (57, 8, 3), (118, 2, 17), (1, 2, 119), (3, 120, 1),
          (1, 1, 1)]


def _phi(shape, rng):
    z, y, x = np.meshgrid(*[np.arange(n) + 0.5 for n in shape], indexing="ij")
    r = np.sqrt((x - 0.4 * shape[2]) ** 2 + (y - 0.5 * shape[1]) ** 2 + (z - 0.5 * shape[0]) ** 2)
    return (r - 0.3 * max(shape)) / max(shape) + 1e-3 * rng.standard_normal(shape)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("flow", ["smooth", "one_sign", "mixed"])
def test_advect_segments_bitwise(cuda, shape, flow):
    rng = np.random.default_rng(11)
    phi = _phi(shape, rng)
    idx = np.indices(shape).sum(0)
    if flow == "smooth":      # regions of either sign, zero stretches between
        vel = [np.sin(0.15 * idx + k) * (np.abs(np.sin(0.07 * idx + k)) > 0.3) for k in range(3)]
    elif flow == "one_sign":
        vel = [np.abs(rng.standard_normal(shape)) * s for s in (1.0, -1.0, 1.0)]
    else:                     # random signs, signed zeros, zeros of phi
        vel = [rng.standard_normal(shape) * rng.integers(0, 2, shape) for _ in range(3)]
        vel = [np.where(rng.random(shape) < 0.1, -0.0, v) for v in vel]
        phi = np.where(rng.random(shape) < 0.1, -0.0, phi)
    spacing = (0.1, 0.25, 1.0 / 3.0)
    want = orc.ls_advect(phi, *vel, 1e-2, spacing, steps=2)
    got = phi.copy()
    with LevelSet(shape, spacing) as ls:
        ls.advect(got, *vel, dt=1e-2, steps=2)
    assert got.tobytes() == want.tobytes()  # the signs of zeros too


@pytest.mark.parametrize("shape", SHAPES[:-1])
def test_redistance_segments(cuda, shape):
    """btn = 0 bit for bit; btn = 1 (sin and cos of two libraries) to 1e-12,
    with cells far outside the band, where the correction is skipped."""
    rng = np.random.default_rng(12)
    h = 0.3 / max(shape)
    phi = _phi(shape, rng)
    for btn in (0, 1):
        want, it_w, _ = orc.ls_redistance(phi, 1.5 * h, 0.1 * h, (h, h, h), btn=btn, max_iter=4)
        got = phi.copy()
        with LevelSet(shape, (h, h, h)) as ls:
            _, it, _ = ls.redistance(got, 1.5 * h, 0.1 * h, btn=btn, max_iter=4)
        assert it == it_w
        if btn == 0:
            np.testing.assert_array_equal(got, want)
        else:
            np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * np.abs(phi).max())


def test_not_finite_values_spread_as_in_the_oracle(cuda):
    """A NaN, an infinity and a huge velocity reach the same cells."""
    rng = np.random.default_rng(13)
    shape, h = (1, 20, 70), 0.1
    phi = _phi(shape, rng)
    u, v, w = (rng.standard_normal(shape) for _ in range(3))
    phi[0, 4, 10], phi[0, 12, 40] = np.nan, np.inf
    u[0, 15, 60], v[0, 3, 50] = np.inf, 1e308
    with np.errstate(all="ignore"):
        want = orc.ls_advect(phi, u, v, w, 1e-3, (h, h, h), steps=1)
    got = phi.copy()
    with LevelSet(shape, (h, h, h)) as ls:
        ls.advect(got, u, v, w, dt=1e-3)
    np.testing.assert_array_equal(got, want)
