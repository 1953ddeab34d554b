"""What gbmg_profile counts where: levels in tiles restrict and prolong inside their
smoother launches, levels in separate launches do not."""
import pytest

from fortrancfd_gb300 import PressurePoisson
from tests import cases

pytestmark = pytest.mark.gpu


def _profile(c):
    with PressurePoisson(c.shape, c.spacing) as s:
        s.ppe_init(c.rho)
        s.set_profiling(True)
        before = s.kernel_launches
        _, st = s.solve(c.b, tol=1e-8)
        prof = {k: n for k, (_, n) in s.profile().items()}
        # (the right-hand side's preparation is not among the classes)
        assert 0 < sum(prof.values()) <= s.kernel_launches - before
        return {k: n / st["cycles"] for k, n in prof.items()}


def test_levels_in_tiles(cuda):
    prof = _profile(cases.config(0))  # 128 x 128 FP64: 128^2, 64^2 and 32^2 in tiles
    assert prof["smooth_fine"] == 2 and prof["smooth_coarse"] == 4 and prof["coarse_solve"] == 1
    for k in ("restrict_fine", "restrict_coarse", "prolong_fine", "prolong_coarse"):
        assert prof[k] == 0


def test_levels_in_separate_launches(cuda):
    prof = _profile(cases.config(1, 8))  # 32^3 FP64: 32^3 and 16^3, then the bottom block
    assert prof["smooth_fine"] == 8 and prof["smooth_coarse"] == 8 and prof["coarse_solve"] == 1
    for k in ("restrict_fine", "restrict_coarse", "prolong_fine", "prolong_coarse"):
        assert prof[k] == 1
