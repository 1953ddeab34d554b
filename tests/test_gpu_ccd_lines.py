"""The two kernels of the compact-difference sweeps at the edges of their
batches: four lanes per line (few lines; eight lines and four points at a time)
and one line per thread (many lines), derivatives bit for bit the oracle's."""
import numpy as np
import pytest

from fortrancfd_gb300 import NSParams, PressurePoisson, curv
from oracle import oracle as orc
from tests.test_gpu_curvature import _check, _phi

pytestmark = pytest.mark.gpu


# line lengths n + 6 with every remainder of 4, line counts off a multiple of
# 8; the last has 19,180 lines in a launch
@pytest.mark.parametrize("shape", [(1, 4, 5), (1, 6, 9), (1, 7, 8), (4, 6, 10), (1, 3, 21),
                                   (64, 96, 64)])
@pytest.mark.parametrize("h", [1.0 / 64, 0.037])
def test_sweeps_match_oracle(cuda, shape, h):
    three = shape[0] > 1
    g = 2
    rng = np.random.default_rng(1)
    phi = _phi(shape)[(slice(1, -1),) * (3 if three else 2)]  # two ghost layers
    if h != 1.0 / 64:  # zero stretches and signed zeros
        phi = np.where(rng.random(phi.shape) < 0.2, -0.0, phi)
        phi[..., :4] = 0.0
    want = orc.ns_curvature(shape, (h, 1.3 * h, 0.7 * h), g, np.ascontiguousarray(phi))
    out = [np.zeros_like(phi) for _ in range(4)]
    with PressurePoisson(shape, (h, 1.3 * h, 0.7 * h)) as pp:
        curv(pp, NSParams(dt=1.0, ghost=g), np.ascontiguousarray(phi), out[0], out[1],
             out[2] if three else None, out[3])
    _check(out, want, three)
