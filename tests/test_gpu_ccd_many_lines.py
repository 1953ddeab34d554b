"""The one-line-per-thread sweep of the compact differences with three ghost layers, as
the time step has them: line lengths of 2 modulo 4, which end the batches of four
points part-way forward and backward.  (Two layers give 0 modulo 4; grids with so
many lines are even along every axis, so there are no others.)"""
import os
import re

import numpy as np
import pytest

import fortrancfd_gb300
from fortrancfd_gb300 import NSParams, PressurePoisson, curv
from oracle import oracle as orc
from tests.test_gpu_curvature import _check, _phi

pytestmark = pytest.mark.gpu

CSRC = os.path.join(os.path.dirname(fortrancfd_gb300.__file__), "csrc")


def _many_lines():
    with open(os.path.join(CSRC, "gbmg_internal.h")) as f:
        return int(re.search(r"kCcdManyLines = (\d+);", f.read()).group(1))


@pytest.mark.parametrize("shape,ghost", [((64, 96, 64), 3), ((96, 64, 128), 3), ((64, 96, 64), 2)])
@pytest.mark.parametrize("h", [1.0 / 64, 0.037])
def test_sweeps_match_oracle(cuda, shape, ghost, h):
    z, y, x = (n + 2 * ghost for n in shape)
    assert y * z + x * z + x * y >= _many_lines()  # the lines of one launch
    assert all((n + 2 * ghost) % 4 == (2 if ghost == 3 else 0) for n in shape)
    rng = np.random.default_rng(2)
    phi = _phi(shape)
    phi = phi if ghost == 3 else np.ascontiguousarray(phi[1:-1, 1:-1, 1:-1])
    if h != 1.0 / 64:  # zero stretches and signed zeros
        phi = np.where(rng.random(phi.shape) < 0.2, -0.0, phi)
        phi[..., :4] = 0.0
    spacing = (h, 1.3 * h, 0.7 * h)
    want = orc.ns_curvature(shape, spacing, ghost, phi)
    out = [np.zeros_like(phi) for _ in range(4)]
    with PressurePoisson(shape, spacing) as pp:
        curv(pp, NSParams(dt=1.0, ghost=ghost), phi, *out)
    _check(out, want, True)
