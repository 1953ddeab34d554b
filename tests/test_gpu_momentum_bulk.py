"""What the momentum kernels leave out (interface terms where delta is zero,
the downwind difference) and where they must not: bit for bit the oracle on
states with rest, signed zeros, parameters outside the fast ranges, and values
that are huge or not finite."""
import numpy as np
import pytest

from fortrancfd_gb300 import PressurePoisson, ns_ab_predictor
from tests.test_gpu_momentum import _oracle_predict, _setup, _state_for_lib

pytestmark = pytest.mark.gpu


def _same(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    return bool(np.all((a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))))


def _check(case, st, prm):
    three = case.shape[0] > 1
    with np.errstate(all="ignore"):
        src, vel = _oracle_predict(case, st, prm)
    s = _state_for_lib(st, three)
    with PressurePoisson(case.shape, case.spacing) as pp:
        ns_ab_predictor(pp, prm, s)
    for c, (k, sk) in enumerate(zip("uvw", ("su", "sv", "sw"))):
        if c == 2 and not three:
            break
        assert _same(s[k], vel[c]), k
        assert _same(s[sk], src[c]), sk


@pytest.mark.parametrize("shape", [(1, 40, 64), (16, 24, 40)])
@pytest.mark.parametrize("extent", [None, (1.0, 0.7, 0.9)])
def test_states_with_rest_and_signed_zeros(cuda, shape, extent):
    case, st, prm = _setup(shape, extent=extent, noise=0.0)
    rng = np.random.default_rng(2)
    for k in ("u", "v", "w"):
        if st[k] is not None:
            st[k][..., : st[k].shape[-1] // 3] = 0.0
            st[k][..., -5:] = -0.0
            st[k] = np.where(rng.random(st[k].shape) < 0.05, -0.0, st[k])
    for k in ("su_old", "sv_old", "sw_old"):
        if st[k] is not None:
            st[k][:, ::3] = 0.0
    _check(case, st, prm)


@pytest.mark.parametrize("change", [dict(mu_12=1.0), dict(re=1e30), dict(re=3.0, we=1e-25),
                                    dict(gravity=(0.0, -0.0, 0.0)), dict(btn_sf=-1.5),
                                    dict(adv_scheme=1)])
def test_parameters(cuda, change):
    case, st, prm = _setup((8, 16, 40))
    for k, v in change.items():
        setattr(prm, k, v)
    _check(case, st, prm)


@pytest.mark.parametrize("shape", [(1, 40, 64), (8, 16, 40)])
def test_huge_and_not_finite_values(cuda, shape):
    """Planted far from the bubble, where the interface terms are zero and
    only their other factors carry the value."""
    case, st, prm = _setup(shape)
    nx = shape[2]
    plants = [("u", 1e300), ("v", -np.inf), ("phi", np.nan), ("phi", 1e308), ("curv", np.inf),
              ("rho", 0.0), ("rho", 1e-308), ("nrm_x", np.nan), ("v", 1e308), ("u", 3e-310),
              ("su_old", 1e-309), ("mu", 1e300)]
    for t, (k, val) in enumerate(plants):
        a = st[k]
        at = (3 + t % (a.shape[0] - 6),) * (a.ndim - 2)
        j = 4 if t % 2 else a.shape[-2] - 6
        a[at + (j, 4 + (t * (nx - 8)) // len(plants))] = val
    _check(case, st, prm)
