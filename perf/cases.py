"""What a user of this package has it do, as cases that can be timed and checked.

A case is a dict of plain values.  "kind" names the call:

  solve       rho_mu + solve from p = 0 on device arrays (the pressure solve)
  host        the same through host arrays (a Fortran host's call)
  project     rho_mu + ppe_solver: right-hand side, solve, velocity correction
  adjoint     the differentiable solve, forward and backward
  advect      one level-set advection step
  redistance  one redistancing call of the level set
  curvature   compact-difference normals and curvature
  momentum    the Adams-Bashforth step: sources, four predictor-projection passes
  step        a restart and one whole time step (mass-preserving level set)

Geometry follows the benchmark's bubbles (smoothed density, ratio 1000, half
width 1.5 cells); pressure solves have a random u*, as there, and transport
and momentum a smooth velocity of a few Fourier modes.
"""
import math

import numpy as np
import torch

from fortrancfd_gb300 import (InterfaceParams, LevelSet, NSParams, PressurePoisson, TwoPhaseStep,
                              curv, ns_ab_solver)
from fortrancfd_gb300.autograd import pressure_solve

F64 = torch.float64
GHOST = 3
RHO_POS, RHO_NEG = 1000.0, 1.0   # outside and inside the bubbles (pressure solves)
RHO_12 = 1e-3                    # the same ratio in the two-phase step's units
MU_12, RE, FR, WE = 1e-2, 1000.0, 0.4096, 1000.0
TOL = 1e-10
ADJOINT_TOL = 1e-8


def _case(name, kind, nx, ny, nz, **kw):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": "mixed",
         "krylov": "none", "bubbles": 1}
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call in earnest: a 2D rising-bubble projection, the
        # reference's own 2D grid size, parity precision
        _case("project2d_128_fp64", "project", 128, 128, 1, precision="fp64"),
        # the headline solve, in the mode that is meant for production
        _case("solve3d_256_mixed", "solve", 256, 256, 256),
        # the same system in the parity form of the reference's multigrid
        _case("solve3d_256_fp64", "solve", 256, 256, 256, precision="fp64"),
        # the largest: many small light bubbles, which need a Krylov method
        _case("solve3d_512_fcg", "solve", 512, 512, 512, krylov="fcg", bubbles=16),
        # a gradient through a solve (design and inverse problems)
        _case("adjoint2d_1024_fgmres", "adjoint", 1024, 1024, 1, krylov="fgmres", bubbles=8),
        # a Fortran host that keeps its arrays in host memory, ragged box
        _case("host3d_160x96x128", "host", 160, 96, 128),
        # interface transport alone: advection on the headline grid,
        # redistancing on an odd box
        _case("advect3d_256", "advect", 256, 256, 256),
        _case("redistance3d_143x127x101", "redistance", 143, 127, 101),
        # normals and curvature of the surface tension, every step
        _case("curvature3d_192x128x256", "curvature", 192, 128, 256),
        # the velocity step around the projection, ragged box
        _case("momentum3d_160x96x128", "momentum", 160, 96, 128),
        # whole time steps: a 2D rising bubble (launches and host work count)
        # and the production 3D grid
        _case("step2d_128x256", "step", 128, 256, 1),
        _case("step3d_256", "step", 256, 256, 256),
    ]


def draw(rng):
    """One more case: any kind, sizes over the listed range (multigrid sizes
    are m 2^k with a product of the m's that the coarsest level takes)."""
    kind = rng.choice(["solve", "host", "project", "adjoint", "advect", "redistance",
                       "curvature", "momentum", "step"])
    two = kind in ("adjoint",) or rng.random() < 0.3
    c = _case("", kind, 1, 1, 1)
    del c["name"]
    if kind in ("advect", "redistance"):   # any size
        hi = (1024 if two else 256) if kind == "advect" else (512 if two else 144)
        c["nx"], c["ny"] = (int(2 ** rng.uniform(math.log2(40), math.log2(hi))) for _ in "xy")
        c["nz"] = 1 if two else int(2 ** rng.uniform(math.log2(24), math.log2(hi)))
        return c
    if two:
        k = rng.choice([4, 5] if kind in ("momentum", "step") else [4, 5, 6, 7])
        c["nx"], c["ny"] = (rng.choice([3, 4, 5, 6, 7, 8]) << k for _ in "xy")
    else:
        k = rng.choice([4, 5, 6])
        m = (2, 3, 4)
        c["nx"], c["ny"], c["nz"] = (rng.choice(m) << k for _ in "xyz")
    if kind == "adjoint":
        c["krylov"] = "fgmres"
        c["bubbles"] = rng.choice([1, 4, 8])
    elif kind in ("solve", "host", "project"):
        c["precision"] = rng.choice(["mixed", "mixed", "fp64"])
        c["krylov"] = rng.choice(["fcg", "fcg", "fgmres", "none"])
        if c["krylov"] != "none":
            c["bubbles"] = rng.choice([1, 2, 4])
    else:
        c["krylov"] = rng.choice(["none", "fcg"]) if kind in ("momentum", "step") else "none"
    return c


# ---- inputs ------------------------------------------------------------------
def _dims(c):
    """(shape (nz, ny, nx), cell width, extents (x, y, z))"""
    shape = (c["nz"], c["ny"], c["nx"])
    short = min(n for n in shape if n > 1)
    h = 1.0 / short
    return shape, h, (c["nx"] * h, c["ny"] * h, c["nz"] * h if c["nz"] > 1 else 1.0)


def _bubbles(c, seed):
    """Seeded bubble centres and radii: one of radius 0.2 with a jittered
    centre, or several small ones that neither overlap nor touch a wall."""
    shape, h, ext = _dims(c)
    three = shape[0] > 1
    rng = np.random.default_rng([seed, 101])
    n = c["bubbles"]
    if n == 1:
        at = np.array([0.5 * ext[0], 0.5 * ext[1], (0.3 if three else 0.5) * ext[2]])
        at[: 3 if three else 2] += rng.uniform(-0.02, 0.02, 3 if three else 2)
        return at[None], np.array([0.2 if three else 0.25])
    lo, hi = (0.03, 0.08) if n == 16 else (0.06, 0.1)
    centres, radii = [], []
    while len(centres) < n:
        r = rng.uniform(lo, hi)
        p = np.array([rng.uniform(r + 0.02, e - r - 0.02) for e in ext])
        if not three:
            p[2] = 0.5
        if all(np.linalg.norm(p - q) > r + s for q, s in zip(centres, radii)):
            centres.append(p)
            radii.append(r)
    return np.array(centres), np.array(radii)


def _coords(c, ghost):
    """Cell centres along z, y, x as broadcastable CUDA tensors (2D: z = 0.5)."""
    shape, h, ext = _dims(c)
    out = []
    for a, n in enumerate(shape):
        if n == 1:
            out.append(torch.full((1, 1, 1), 0.5, dtype=F64, device="cuda"))
            continue
        x = (torch.arange(n + 2 * ghost, dtype=F64, device="cuda") - ghost + 0.5) * h
        out.append(x.reshape([-1 if b == a else 1 for b in range(3)]))
    return out


def _phi(c, seed, ghost=0):
    """Signed distance to the bubbles, negative inside."""
    Z, Y, X = _coords(c, ghost)
    phi = None
    for p, r in zip(*_bubbles(c, seed)):
        d = torch.sqrt((X - p[0]) ** 2 + (Y - p[1]) ** 2 + (Z - p[2]) ** 2) - r
        phi = d if phi is None else torch.minimum(phi, d)
    return phi.contiguous()


def _smooth(c, seed, ghost, amplitude, which):
    """A smooth field of four random Fourier modes."""
    Z, Y, X = _coords(c, ghost)
    rng = np.random.default_rng([seed, 202, which])
    f = 0.0
    for _ in range(4):
        k, ph, a = rng.integers(1, 4, 3), rng.uniform(0, 2 * np.pi, 3), rng.standard_normal()
        z = torch.sin(k[2] * np.pi * Z + ph[2]) if c["nz"] > 1 else 1.0
        f = f + a * (torch.sin(k[0] * np.pi * X + ph[0]) * torch.sin(k[1] * np.pi * Y + ph[1]) * z)
    return (amplitude * f).contiguous()


def _random_velocity(c, seed):
    """u* ~ N(0, 1) on the interior faces, 0 on the walls."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 * int(seed) + 7)
    nz, ny, nx = _dims(c)[0]
    u, v, w = (torch.randn(s, generator=g, device="cuda", dtype=F64)
               for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)))
    u[..., 0] = u[..., -1] = 0.0
    v[:, 0] = v[:, -1] = 0.0
    w[0] = w[-1] = 0.0
    return u, v, (w if nz > 1 else None)


def _divergence(u, v, w, h, dt):
    d = (u[..., 1:] - u[..., :-1]) / h + (v[:, 1:] - v[:, :-1]) / h
    return (d if w is None else d + (w[1:] - w[:-1]) / h) / dt


def _walls(fields, g):
    """No-slip ghosts of padded face velocities (velbc): the values mirrored
    with a minus sign, the wall-normal face 0."""
    for ax in range(len(fields)):
        for comp, f in enumerate(fields):
            a = f.movedim(f.ndim - 1 - ax, -1)
            n = a.shape[-1] - 2 * g
            own = comp == ax
            for m in range(1, g + 1):
                a[..., g - m] = -a[..., g + (m - 1 if own else m) - 1]
                a[..., g + n + m - 1] = -a[..., g + (n - m if own else n + 1 - m) - 1]
            if own:
                a[..., g - 1] = 0.0
                a[..., g + n - 1] = 0.0
    return fields


def _heaviside(phi, eps):
    """(H, dH/dphi) with half width eps."""
    x = phi / eps
    h = 0.5 * (1.0 + x + torch.sin(np.pi * x) / np.pi)
    h = torch.where(x > 1 - 1e-12, 1.0, torch.where(x < -1 + 1e-12, 0.0, h)).clamp(0.0, 1.0)
    d = torch.where(x.abs() < 1 - 1e-12, 0.5 * (1.0 + torch.cos(np.pi * x)) / eps, 0.0)
    return h, d


def _ns(c):
    """The momentum step's parameters, dt below its explicit viscous limit."""
    shape, h, _ = _dims(c)
    three = shape[0] > 1
    nu = MU_12 / RHO_12 / RE
    return NSParams(dt=0.8 * h * h / ((6 if three else 4) * nu), re=RE, fr=FR, we=WE, mu_12=MU_12,
                    gravity=(0.0, 0.0, -1.0) if three else (0.0, -1.0, 0.0), btn_g=1.0,
                    btn_sf=1.0, ghost=GHOST, iterations=4, p_tol=TOL)


def _squeeze(c, a):
    """Padded arrays have no z axis in 2D."""
    return a if c["nz"] > 1 else a[0]


def _momentum_inputs(c, seed):
    """Padded fields of the momentum step: a bubble and smooth velocities."""
    _, h, _ = _dims(c)
    three = c["nz"] > 1
    phi = _phi(c, seed, GHOST)
    heavy, delta = _heaviside(phi, 1.5 * h)
    f = {"phi": phi, "delta": delta, "rho": heavy + RHO_12 * (1 - heavy),
         "mu": heavy + MU_12 * (1 - heavy)}
    for i, k in enumerate(("u", "v", "w", "su_old", "sv_old", "sw_old")):
        f[k] = None if not three and i % 3 == 2 else _smooth(c, seed, GHOST, 0.1, i)
    f = {k: None if a is None else _squeeze(c, a).contiguous() for k, a in f.items()}
    _walls([f[k] for k in "uvw" if f[k] is not None], GHOST)
    return f


def _inner(c, a):
    """(nz, ny, nx) interior of a padded cell array."""
    s = slice(GHOST, -GHOST)
    return a[s, s, s] if c["nz"] > 1 else a[s, s][None]


def _solver(c, max_cycles=400):
    shape, h, _ = _dims(c)
    return PressurePoisson(shape, (h, h, h), precision=c["precision"], krylov=c["krylov"],
                           max_cycles=max_cycles)


def prepare(case, seed):
    c = case
    shape, h, _ = _dims(c)
    s = {"case": c, "h": h}
    kind = c["kind"]
    if kind in ("solve", "host", "project", "adjoint"):
        s["pp"] = _solver(c)
        s["phi"] = _phi(c, seed)
        vel = _random_velocity(c, seed)
        s["dt"] = 1e-3
        if kind == "project":
            s["vel0"] = vel
            s["vel"] = [None if a is None else a.clone() for a in vel]
        else:
            s["b"] = _divergence(*vel, h, s["dt"])
        s["p"] = torch.zeros(shape, dtype=F64, device="cuda")
        if kind == "host":   # pinned arrays, as a host code keeps them
            for k in ("phi", "b", "p"):
                t = s.pop(k)
                s[k + "_t"] = torch.empty(shape, dtype=F64, pin_memory=True).copy_(t)
                s[k] = s[k + "_t"].numpy()
        if kind == "adjoint":
            s["target"] = _smooth(c, seed, 0, 10.0, 9)
        return s
    if kind in ("advect", "redistance"):
        s["ls"] = LevelSet(shape, (h, h, h))
        s["phi0"] = _phi(c, seed)
        if kind == "redistance":   # a level set that transport has distorted
            s["phi0"] = s["phi0"] * (1.0 + _smooth(c, seed, 0, 0.2, 5).clamp(-0.5, 0.5))
        else:
            s["vel"] = [_smooth(c, seed, 0, 1.0, i) if i < (3 if c["nz"] > 1 else 2) else None
                        for i in range(3)]
            s["dt"] = 0.1 * h
        s["phi"] = s["phi0"].clone()
        return s
    ns = s["ns"] = _ns(c)
    if kind == "curvature":
        s["pp"] = _solver(c)
        s["phi"] = _squeeze(c, _phi(c, seed, GHOST)).contiguous()
        s["out"] = [torch.zeros_like(s["phi"]) for _ in range(4)]
        return s
    f = _momentum_inputs(c, seed)
    if kind == "step":
        itf = InterfaceParams(ls_wid=1.5 * h, rho_12=RHO_12, rdt=0.25 * h, redis_every=5, method=2)
        s["ts"] = TwoPhaseStep(shape, (h, h, h), ns, itf, precision=c["precision"],
                               krylov=c["krylov"])
        s["init"] = {k: f[k] for k in ("phi", "u", "v", "w")}
        return s
    s["pp"] = _solver(c)
    s["rho_now"] = _inner(c, f["rho"]).contiguous()
    grads = [torch.empty_like(f["phi"]) for _ in range(4)]
    curv(s["pp"], ns, f["phi"], grads[0], grads[1], grads[2], grads[3])
    st = {k: f[k] for k in ("rho", "mu", "delta", "phi", "su_old", "sv_old", "sw_old")}
    st.update(u_old=f["u"], v_old=f["v"], w_old=f["w"], nrm_x=grads[0], nrm_y=grads[1],
              nrm_z=grads[2] if c["nz"] > 1 else None, curv=grads[3])
    for k in ("u", "v", "w", "su", "sv", "sw"):
        st[k] = None if f[k[-1]] is None else torch.zeros_like(f["phi"])
    st["p"] = torch.zeros(shape if c["nz"] > 1 else shape[1:], dtype=F64, device="cuda")
    s["state"] = st
    return s


# ---- one pass ----------------------------------------------------------------
def run(state):
    s, c = state, state["case"]
    kind, eps = c["kind"], 1.5 * state["h"]
    if kind == "solve":
        s["pp"].rho_mu(s["phi"], eps, RHO_POS, RHO_NEG)
        s["p"].zero_()
        s["pp"].solve(s["b"], s["p"], tol=TOL)
        return s["p"]
    if kind == "host":
        s["pp"].rho_mu(s["phi"], eps, RHO_POS, RHO_NEG)
        s["p"].fill(0.0)
        s["pp"].solve(s["b"], s["p"], tol=TOL)
        return s["p"]
    if kind == "project":
        for a, b in zip(s["vel"], s["vel0"]):
            if a is not None:
                a.copy_(b)
        s["p"].zero_()
        s["pp"].rho_mu(s["phi"], eps, RHO_POS, RHO_NEG)
        s["pp"].ppe_solver(*s["vel"], s["dt"], tol=TOL, p=s["p"])
        return [s["p"]] + [a for a in s["vel"] if a is not None]
    if kind == "adjoint":
        phi = s["phi"].clone().requires_grad_(True)
        b = s["b"].clone().requires_grad_(True)
        p = pressure_solve(phi, b, s["pp"], eps, RHO_POS, RHO_NEG, TOL, ADJOINT_TOL)
        (0.5 * ((p - s["target"]) ** 2).sum()).backward()
        return {"p": p.detach(), "grad_b": b.grad, "grad_phi": phi.grad}
    if kind == "advect":
        s["phi"].copy_(s["phi0"])
        return s["ls"].advect(s["phi"], *s["vel"], dt=s["dt"], steps=1)
    if kind == "redistance":
        s["phi"].copy_(s["phi0"])
        phi, iterations, _ = s["ls"].redistance(s["phi"], eps, 0.25 * s["h"], RHO_12, btn=1)
        return [phi, iterations]
    if kind == "curvature":
        curv(s["pp"], s["ns"], s["phi"], *s["out"])
        return s["out"] if c["nz"] > 1 else [s["out"][0], s["out"][1], s["out"][3]]
    if kind == "momentum":
        st = s["state"]
        for k in "uvw":   # the time loop's switch leaves the old velocity here
            if st[k] is not None:
                st[k].copy_(st[k + "_old"])
        st["p"].zero_()
        s["pp"].ppe_init(s["rho_now"])
        ns_ab_solver(s["pp"], s["ns"], st)
        return {k: st[k] for k in ("u", "v", "w", "su", "sv", "sw", "p") if st[k] is not None}
    ts, z = s["ts"], s["init"]
    ts.load(z["phi"], z["u"], z["v"], z["w"],
            p=torch.zeros(ts.p.shape, dtype=F64, device="cuda"))
    ts.step()
    return dict({k: ts.now[k] for k in ("phi", "u", "v", "w", "rho", "curv")
                 if ts.now[k] is not None}, p=ts.p)


def work(case):
    """Bytes: every input read once and every output written once.  Operations:
    one sweep over the unknowns per unit of a pass that no method avoids (the
    stencil of one residual; the reconstructions of every face and stage)."""
    n = case["nx"] * case["ny"] * case["nz"]
    d = 3 if case["nz"] > 1 else 2
    kind = case["kind"]
    if kind in ("solve", "host"):
        return {"bytes": 24.0 * n, "flops": 20.0 * n}
    if kind == "project":
        return {"bytes": (16.0 + 16.0 * d) * n, "flops": 30.0 * n}
    if kind == "adjoint":
        return {"bytes": 48.0 * n, "flops": 60.0 * n}
    if kind == "advect":
        return {"bytes": (16.0 + 8.0 * d) * n, "flops": 3.0 * 160.0 * d * n}
    if kind == "redistance":   # 13 iterations of three stages at this pseudo-time step
        return {"bytes": 16.0 * n, "flops": 13.0 * 3.0 * 160.0 * d * n}
    if kind == "curvature":
        return {"bytes": (16.0 + 8.0 * d) * n, "flops": 40.0 * (6 if d == 3 else 3) * n}
    if kind == "momentum":   # old velocity and sources, six cell fields; new velocity, source, p
        return {"bytes": (8.0 * (4 * d + 5 + d) + 8.0) * n, "flops": (70.0 + 4 * 45.0) * d * n}
    return {"bytes": 8.0 * (4 * d + 12) * n, "flops": (3 * 160.0 + 4 * 45.0 + 70.0) * d * n}


# ---- the same in plain 64-bit torch -------------------------------------------
def _face_sum(rho):
    """rho_i + rho_nb on the interior faces of each axis (x, y, z)."""
    out = [rho[..., 1:] + rho[..., :-1], rho[:, 1:] + rho[:, :-1]]
    return out + ([rho[1:] + rho[:-1]] if rho.shape[0] > 1 else [])


def _poisson(coef, b, limit=1500):
    """The mean-free p with sum_f coef_f (p_nb - p) = b - mean(b): conjugate
    gradients, preconditioned by the constant-coefficient operator (cosine
    transforms along each axis)."""
    shape = b.shape
    mats, lam = [], 0.0
    for a, n in enumerate(shape):
        if n == 1:
            mats.append(None)
            continue
        i = torch.arange(n, dtype=F64, device=b.device)
        C = torch.cos(np.pi * i[:, None] * (i[None] + 0.5) / n) * math.sqrt(2.0 / n)
        C[0] /= math.sqrt(2.0)
        mats.append(C)
        lam = lam + (2 - 2 * torch.cos(np.pi * i / n)).reshape([-1 if q == a else 1 for q in range(3)])
    lam[0, 0, 0] = 1.0

    def along(C, x, a):
        return (C @ x.movedim(a, 0).reshape(x.shape[a], -1)).reshape(
            x.movedim(a, 0).shape).movedim(0, a)

    def precondition(r):
        for a, C in enumerate(mats):
            r = r if C is None else along(C, r, a)
        r = r / lam
        r[0, 0, 0] = 0.0
        for a, C in enumerate(mats):
            r = r if C is None else along(C.T, r, a)
        return r.contiguous()

    def apply(p):   # -A p
        q = torch.zeros_like(p)
        for ax, cf in zip((2, 1, 0), coef):
            n = p.shape[ax]
            f = cf * (p.narrow(ax, 1, n - 1) - p.narrow(ax, 0, n - 1))
            q.narrow(ax, 0, n - 1).sub_(f)
            q.narrow(ax, 1, n - 1).add_(f)
        return q

    r = -(b - b.mean())
    x = torch.zeros_like(b)
    stop = 1e-14 * float(r.norm())
    z = precondition(r)
    d, rz, best, flat = z.clone(), float((r * z).sum()), math.inf, 0
    for _ in range(limit):
        q = apply(d)
        a = rz / float((d * q).sum())
        x += a * d
        r -= a * q
        size = float(r.norm())
        best, flat = (size, 0) if size < 0.5 * best else (best, flat + 1)
        if size < stop or flat > 200:
            break
        z = precondition(r)
        new = float((r * z).sum())
        d = z + (new / rz) * d
        rz = new
    return x - x.mean()


def _project(rho, vel, h, dt):
    """p and the corrected face velocities (u, v(, w)) of one projection."""
    rs = _face_sum(rho)
    w = vel[2] if len(vel) > 2 else None
    p = _poisson([2.0 / s / (h * h) for s in rs], _divergence(vel[0], vel[1], w, h, dt))
    for ax, s, f in zip((2, 1, 0), rs, vel):
        n = p.shape[ax]
        f.narrow(ax, 1, n - 1).sub_(dt * (p.narrow(ax, 1, n - 1) - p.narrow(ax, 0, n - 1)) / h
                                    / (0.5 * s))
    return p


def _at(f, ax, lo, n):
    """f at indices lo .. lo + n - 1 of axis ax, clamped to the grid."""
    i = torch.arange(lo, lo + n, device=f.device).clamp(0, f.shape[ax] - 1)
    return f.index_select(ax, i)


def _weno(g, eps):
    """Left-biased fifth-order WENO-JS value at the face right of g[2]."""
    b = [13 * (g[k] - 2 * g[k + 1] + g[k + 2]) ** 2 + 3 * t ** 2 for k, t in
         enumerate((g[0] - 4 * g[1] + 3 * g[2], g[1] - g[3], 3 * g[2] - 4 * g[3] + g[4]))]
    a = [q / (eps + x) ** 2 for q, x in zip((1.0, 6.0, 3.0), b)]
    s = a[0] + a[1] + a[2]
    return (a[0] * (2 * g[0] - 7 * g[1] + 11 * g[2]) + a[1] * (-g[1] + 5 * g[2] + 2 * g[3])
            + a[2] * (2 * g[2] + 5 * g[3] - g[4])) / (6 * s)


def _advect(phi, vel, h, dt):
    def rate(f):
        out = torch.zeros_like(f)
        for ax, u in zip((2, 1, 0), vel):
            n = f.shape[ax]
            gp, gm = u.clamp(min=0) * f, u.clamp(max=0) * f
            face = _weno([_at(gp, ax, m - 3, n + 1) for m in range(5)], 1e-13)
            face += _weno([_at(gm, ax, 2 - m, n + 1) for m in range(5)], 1e-13)
            out -= (face.narrow(ax, 1, n) - face.narrow(ax, 0, n)) / h
        return out

    phi = phi.clone()
    l1 = rate(phi)
    phi += dt * l1
    l2 = rate(phi)
    phi += dt * (l2 - 3 * l1) / 4
    return phi + dt * (8 * rate(phi) - l1 - l2) / 12


def _redistance(phi, eps, rdt, h):
    three = phi.shape[0] > 1
    axes = (2, 1, 0) if three else (2, 1)
    sign = 2 * _heaviside(phi, eps)[0] - 1

    def gradient(f):
        sq = 0.0
        for ax in axes:
            n = f.shape[ax]
            d = (f.narrow(ax, 1, n - 1) - f.narrow(ax, 0, n - 1)) / h
            d = torch.cat([torch.zeros_like(d.narrow(ax, 0, 1)), d], ax)   # backward difference
            g = [_at(d, ax, m - 2, n) for m in range(6)]
            right, left = _weno(g[:0:-1], 1e-10), _weno(g[:5], 1e-10)
            t = torch.where(sign >= 0, torch.maximum(-right.clamp(max=0), left.clamp(min=0)),
                            torch.maximum(right.clamp(min=0), -left.clamp(max=0)))
            sq = sq + t * t
        return torch.sqrt(sq)

    def block(x):   # weighted 3^d block sum, clamped at the walls
        s = x
        for ax in axes:
            n = x.shape[ax]
            s = sum(_at(s, ax, m, n) for m in (-1, 0, 1))
        return (51.0 if three else 16.0) * x + s

    def rate(f):
        g = gradient(f)
        hv, dl = _heaviside(f, eps)
        lam = (2 * (1 - RHO_12) * hv + RHO_12) * dl if three else dl
        a, b = block(lam * sign * (g - 1)), block(g * dl * lam)
        s1 = torch.where(b.abs() > 1e-12, a / b * dl, 0.0)
        return (sign - s1) * g - sign

    phi, time, it = phi.clone(), 0.0, 0
    while True:
        it += 1
        time += rdt
        old = phi.clone()
        l1 = rate(phi)
        phi -= rdt * l1
        l2 = rate(phi)
        phi -= rdt * (l2 - 3 * l1) / 4
        phi -= rdt * (8 * rate(phi) - l1 - l2) / 12
        if time > 3 * h or float((phi - old).abs().max()) <= (1e-5 if three else 1e-8):
            return phi, it


def _ccd(n, h, dev):
    """Matrices D1, D2 of the combined compact differences on a line of n points."""
    M, B = np.eye(2 * n), np.zeros((2 * n, n))
    for i in range(1, n - 1):
        M[i, [i - 1, i + 1, n + i - 1, n + i + 1]] = 7 / 16, 7 / 16, h / 16, -h / 16
        M[n + i, [i - 1, i + 1, n + i - 1, n + i + 1]] = -9 / 8 / h, 9 / 8 / h, -1 / 8, -1 / 8
        B[i, [i - 1, i + 1]] = -15 / 16 / h, 15 / 16 / h
        B[n + i, [i - 1, i, i + 1]] = 3 / h ** 2, -6 / h ** 2, 3 / h ** 2
    for i, o, s in ((0, 1, 1.0), (n - 1, -1, -1.0)):
        M[i, [i + o, n + i + o]] = 2.0, -s * h
        M[n + i, [i + o, n + i + o]] = -s * 2.5 / h, 8.5
        B[i, [i, i + o, i + 2 * o]] = -3.5 * s / h, 4.0 * s / h, -0.5 * s / h
        B[n + i, [i, i + o, i + 2 * o, i + 3 * o]] = np.array([34 / 3, -83 / 4, 10, -7 / 12]) / h ** 2
    D = torch.from_numpy(np.linalg.solve(M, B)).to(dev)
    return D[:n], D[n:]


def _line(f, ax, h):
    """(f', f'') along axis ax."""
    x = f.movedim(ax, 0)
    return tuple((D @ x.reshape(x.shape[0], -1)).reshape(x.shape).movedim(0, ax)
                 for D in _ccd(x.shape[0], h, f.device))


def _clamped(a):
    """Zero-gradient ghosts of a padded array, in place."""
    for ax in range(a.ndim):
        n = a.shape[ax]
        a.narrow(ax, 0, GHOST).copy_(a.narrow(ax, GHOST, 1).expand_as(a.narrow(ax, 0, GHOST)))
        a.narrow(ax, n - GHOST, GHOST).copy_(
            a.narrow(ax, n - GHOST - 1, 1).expand_as(a.narrow(ax, 0, GHOST)))
    return a


def _curvature(phi, h):
    """Gradient (x, y(, z)) and curvature of a padded level set."""
    ax = list(range(phi.ndim))[::-1]   # x, y(, z)
    first = [_line(phi, a, h) for a in ax]
    fx, fy = first[0][0], first[1][0]
    fxx, fyy = first[0][1], first[1][1]
    fxy = _line(fx, ax[1], h)[0]
    if phi.ndim == 2:
        num = fyy * fx ** 2 + fxx * fy ** 2 - 2 * fxy * fx * fy
        sq = fx ** 2 + fy ** 2 + 1e-12
    else:
        fz, fzz = first[2]
        fxz, fyz = _line(fx, ax[2], h)[0], _line(fy, ax[2], h)[0]
        num = ((fyy + fzz) * fx ** 2 + (fxx + fzz) * fy ** 2 + (fxx + fyy) * fz ** 2
               - 2 * (fxy * fx * fy + fxz * fx * fz + fyz * fy * fz))
        sq = fx ** 2 + fy ** 2 + fz ** 2 + 1e-12
    return [_clamped(a.contiguous()) for a in [f[0] for f in first] + [num / sq ** 1.5]]


def _sh(a, *off):
    """Interior of a padded array displaced by off = (x, y, z) cells."""
    off = list(off) + [0] * (a.ndim - len(off))
    return a[tuple(slice(GHOST + o, a.shape[q] - GHOST + o)
                   for q, o in enumerate(off[:a.ndim][::-1]))]


def _unit(a, s=1):
    return tuple(s if b == a else 0 for b in range(3))


def _plus(p, q):
    return tuple(a + b for a, b in zip(p, q))


def _momentum(f, ns, h, rho_now, p_shape):
    """The whole momentum step on padded fields f (old fields, normals, curv);
    returns the new velocity and sources (padded) and p."""
    dim = f["phi"].ndim
    names = "uvw"[:dim]
    old = [f[k] for k in names]
    dt = ns.dt
    diff = []
    for a in range(dim):
        e = _unit(a)
        mean = lambda x: 0.5 * (_sh(x) + _sh(x, *e))  # noqa: E731
        rho, mu, delta = mean(f["rho"]), mean(f["mu"]), mean(f["delta"])
        t = 0.0
        for b in range(dim):
            o = _unit(b)
            lap = (_sh(old[a], *o) - 2 * _sh(old[a]) + _sh(old[a], *_unit(b, -1))) / h ** 2
            t = t + mu / rho * lap / ns.re
            # delta (dphi/db) (du_a/db + du_b/da) of the interface viscosity
            if a == b:
                dphi = (_sh(f["phi"], *e) - _sh(f["phi"])) / h
                rate = 2 * 0.5 * (_sh(old[a], *e) - _sh(old[a], *_unit(a, -1))) / h
            else:
                up, dn = _unit(b), _unit(b, -1)
                dphi = 0.25 * (_sh(f["phi"], *_plus(e, up)) - _sh(f["phi"], *_plus(e, dn))
                               + _sh(f["phi"], *up) - _sh(f["phi"], *dn)) / h
                rate = 0.5 * (_sh(old[a], *up) - _sh(old[a], *dn)) / h
                rate = rate + 0.5 * (_sh(old[b], *e) - _sh(old[b]) + _sh(old[b], *_plus(e, dn))
                                     - _sh(old[b], *dn)) / h
            t = t + (1 - ns.mu_12) * delta * dphi * rate / (rho * ns.re)
        t = t + ns.gravity[a] * ns.btn_g / ns.fr
        t = t - ns.btn_sf * mean(f["curv"]) * delta * mean(f["nrm_" + "xyz"[a]]) / (ns.we * rho)
        diff.append(t)
    now = [x.clone() for x in old]
    src = [torch.zeros_like(x) for x in old]
    inner = (slice(GHOST, -GHOST),) * dim
    for _ in range(ns.iterations):
        tmp = [x.clone() for x in now]
        for a in range(dim):
            e, adv = _unit(a), 0.0
            for b in range(dim):
                if a == b:
                    c = _sh(tmp[a])
                else:
                    dn = _unit(b, -1)
                    c = 0.25 * (_sh(tmp[b]) + _sh(tmp[b], *dn) + _sh(tmp[b], *e)
                                + _sh(tmp[b], *_plus(e, dn)))
                fld = old[a]
                fp = 0.5 * (-_sh(fld, *_unit(b, 2)) + 4 * _sh(fld, *_unit(b)) - 3 * _sh(fld)) / h
                fm = 0.5 * (_sh(fld, *_unit(b, -2)) - 4 * _sh(fld, *_unit(b, -1)) + 3 * _sh(fld)) / h
                adv = adv - torch.where(c > 0, c * fm, c * fp)
            s = adv + diff[a]
            src[a][inner] = s
            now[a][inner] = _sh(old[a]) + dt * (1.5 * s - 0.5 * _sh(f["s" + names[a] + "_old"]))
        _walls(now, GHOST)
        faces = []
        for a, x in enumerate(now):   # faces 0 .. n of axis a, interior in the others
            q = x.ndim - 1 - a
            v = x[tuple(slice(GHOST - (b == q), -GHOST) for b in range(dim))]
            faces.append(v if dim == 3 else v[None])
        p = _project(rho_now, faces, h, dt)
        _walls(now, GHOST)
    return now, src, p.reshape(p_shape)


def _mass(phi, h, eps):
    """ls_mv's mass of a padded level set."""
    hv = _heaviside(phi[(slice(GHOST, -GHOST),) * phi.ndim], eps)[0]
    return float(((hv + RHO_12 * (1 - hv)) * hv).sum()) * h ** phi.ndim


def _step(c, z, ns, h):
    """TwoPhaseStep.load and one step of it (no redistancing in the first)."""
    eps = 1.5 * h
    dim = 3 if c["nz"] > 1 else 2
    inner = (slice(GHOST, -GHOST),) * dim
    phi = z["phi"].clone()
    f = {"phi": z["phi"], "u": z["u"], "v": z["v"], "w": z["w"]}
    hv, f["delta"] = _heaviside(phi, eps)
    f["rho"], f["mu"] = hv + RHO_12 * (1 - hv), hv + MU_12 * (1 - hv)
    g = _curvature(phi, h)
    f["nrm_x"], f["nrm_y"], f["curv"] = g[0], g[1], g[-1]
    f["nrm_z"] = g[2] if dim == 3 else None
    vel = []
    for a, k in enumerate("uvw"[:dim]):
        n = 0.5 * (_sh(z[k], *_unit(a, -1)) + _sh(z[k]))
        vel.append(n if dim == 3 else n[None])
        f["s" + k + "_old"] = torch.zeros_like(phi)
    mass = _mass(phi, h, eps)
    box = phi[inner] if dim == 3 else phi[inner][None]
    phi[inner] = _advect(box, vel, h, ns.dt).reshape(phi[inner].shape)
    _clamped(phi)
    for _ in range(2):   # mass_preserving_level_set
        size = torch.sqrt(sum(_line(phi, a, h)[0] ** 2 for a in range(dim)))[inner]
        hv, dl = _heaviside(phi[inner], eps)
        den = float((dl ** 2 * size * (2 * (1 - RHO_12) * hv + RHO_12)).sum()) * h ** dim
        phi[inner] += (mass - _mass(phi, h, eps)) / den * dl * size
        _clamped(phi)
    hv = _heaviside(phi, eps)[0]
    rho = hv + RHO_12 * (1 - hv)
    shape = _dims(c)[0]
    now, _, p = _momentum(f, ns, h, _inner(c, rho).contiguous(), shape if dim == 3 else shape[1:])
    return dict(zip("uvw", now), phi=phi, rho=rho, curv=_curvature(phi, h)[-1], p=p)


def exact(case, seed):
    c = case
    shape, h, _ = _dims(c)
    n, kind, eps = math.prod(shape), c["kind"], 1.5 * h
    # the 512^3 solve and whole 3D steps and momentum steps above two million
    # cells (four or more solves) take longer than is worth waiting for
    if n > (1 << 24) or (kind in ("momentum", "step") and n > (1 << 21)):
        return None
    if kind in ("solve", "host", "project", "adjoint"):
        phi, vel = _phi(c, seed), [a for a in _random_velocity(c, seed) if a is not None]
        hv, dl = _heaviside(phi, eps)
        rho = RHO_POS * hv + RHO_NEG * (1 - hv)
        if kind == "project":
            p = _project(rho, vel, h, 1e-3)
            return [p] + vel
        rs = _face_sum(rho)
        b = _divergence(vel[0], vel[1], vel[2] if len(vel) > 2 else None, h, 1e-3)
        coef = [2.0 / s / (h * h) for s in rs]
        p = _poisson(coef, b)
        if kind != "adjoint":
            return p
        lam = _poisson(coef, p - _smooth(c, seed, 0, 10.0, 9))
        grad = torch.zeros_like(p)
        for ax, s in zip((2, 1, 0), rs):
            m = p.shape[ax]
            hi, lo = (lambda x: x.narrow(ax, 1, m - 1)), (lambda x: x.narrow(ax, 0, m - 1))
            t = (hi(lam) - lo(lam)) * (hi(p) - lo(p)) * (-2.0 / s ** 2 / (h * h))
            hi(grad).add_(t)
            lo(grad).add_(t)
        return {"p": p, "grad_b": lam, "grad_phi": grad * (RHO_POS - RHO_NEG) * dl}
    if kind == "advect":
        return _advect(_phi(c, seed),
                       [_smooth(c, seed, 0, 1.0, i) for i in range(3 if c["nz"] > 1 else 2)],
                       h, 0.1 * h)
    if kind == "redistance":
        phi = _phi(c, seed) * (1.0 + _smooth(c, seed, 0, 0.2, 5).clamp(-0.5, 0.5))
        return list(_redistance(phi, eps, 0.25 * h, h))
    if kind == "curvature":
        return _curvature(_squeeze(c, _phi(c, seed, GHOST)).contiguous(), h)
    ns = _ns(c)
    f = _momentum_inputs(c, seed)
    if kind == "step":
        return _step(c, f, ns, h)
    g = _curvature(f["phi"], h)
    f["nrm_x"], f["nrm_y"], f["curv"] = g[0], g[1], g[-1]
    f["nrm_z"] = g[2] if c["nz"] > 1 else None
    now, src, p = _momentum(f, ns, h, _inner(c, f["rho"]).contiguous(),
                            shape if c["nz"] > 1 else shape[1:])
    return dict(zip("uvw", now), p=p, **{"s" + k: s for k, s in zip("uvw", src)})
