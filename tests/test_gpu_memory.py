"""The stored diagonals of an FP64 handle are kept once, and only where memory is
plentiful: with little memory free a handle is as large as its other arrays, a
later allocation that does not fit takes theirs, and the iterates keep their bits."""
import numpy as np
import pytest
import torch

from fortrancfd_gb300 import NSParams, PressurePoisson, curv, inputs
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPE = (192, 192, 192)
CELL = 8 * 192 ** 3   # an array of the finest level
SLACK = 48 << 20      # driver granularity and the small arrays


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    """Take all but `leave` bytes of the device's memory, to the allocator's 2 MiB."""
    held = []
    while _free() - leave > (32 << 20):
        held.append(torch.empty(min(_free() - leave, 32 << 30), dtype=torch.uint8, device="cuda"))
    return held


def _case(cuda):
    case = inputs.custom(SHAPE, radii=(0.2,))
    phi = torch.from_numpy(inputs.level_set(case)).to(cuda)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    b = torch.randn(SHAPE, generator=g, device="cuda", dtype=torch.float64)
    return case, phi, b - b.mean()


def _solve(case, phi, b, krylov, after=lambda s: None):
    """(bytes that the handle takes, the solution as bytes)"""
    before = _free()
    with PressurePoisson(case.shape, case.spacing, krylov=krylov, max_cycles=60) as s:
        size = before - _free()
        s.rho_mu(phi, case.eps, 1000.0, 1.0)
        s.solve(b, tol=1e-8)
        after(s)
        return size, s.solve(b, tol=1e-8)[0].cpu().numpy().tobytes()


@pytest.mark.parametrize("krylov", ["none", "fcg"])
def test_diagonal_once_or_not_at_all(cuda, krylov):
    case, phi, b = _case(cuda)
    _solve(case, phi, b, krylov)  # (the kernels' code is loaded)
    plenty, want = _solve(case, phi, b, krylov)
    # coefficients, 1/diagonal, b, p, rho; the coarse levels an eighth and so on
    # of six arrays; five Krylov vectors
    bare = (7 + 6 / 7 + (5 if krylov == "fcg" else 0)) * CELL
    diagonals = 8 / 7 * CELL
    assert bare + diagonals - SLACK < plenty < bare + diagonals + SLACK
    held = _fill(int(bare + 4 * diagonals))
    try:
        short, got = _solve(case, phi, b, krylov)
    finally:
        del held
        torch.cuda.empty_cache()
    assert bare - SLACK < short < bare + SLACK
    assert got == want


def test_diagonals_make_room(cuda):
    case, phi, b = _case(cuda)
    prm = NSParams(dt=1.0, ghost=2)
    pad = np.zeros(orc.padded_shape(SHAPE, 2))
    out = [np.zeros_like(pad) for _ in range(4)]
    need = []

    def curvature(s):
        before = _free()
        curv(s, prm, pad, *out)
        need.append(before - _free())

    _solve(case, phi, b, "none", curvature)
    _, want = _solve(case, phi, b, "none", curvature)
    held = []

    def short_of_memory(s):
        held.extend(_fill(need[-1] - CELL // 2))  # half of the finest diagonal is missing
        assert _free() < need[-1]
        curv(s, prm, pad, *out)

    try:
        _, got = _solve(case, phi, b, "none", short_of_memory)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert got == want
