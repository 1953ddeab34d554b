// Level-set transport on sm_103a: the advection step of the reference's
// interface solver, level_set_rk3_solver ("Two phase flows/newOpenMP/2D/src/
// interface_solver/level_set_rk3_solver.f90:1-186"; 3D "Two phase flows/
// newOpenMP/3D+IBM/src/interface_solver/level_set_rk3_solver.f90:1-215").
//
// phi_t + div(u phi) = 0 with the cell-centred velocity: the flux is split
// into u+ phi and u- phi (level_set_rk3_source_setup), each part is
// reconstructed at every face by WENO-JS (wenojs_flux_split, EPS = 1e-13) --
// u+ phi from the five cells left of the face, u- phi from the five cells
// right of it -- with zero-gradient ghosts (bc: an index outside the grid
// reads the nearest boundary cell), and three stages of SSP-RK3 in the
// reference's incremental form advance phi.  nz = 1 is the 2D solver.
//
// The faces are reconstructed once each (k_ls_faces, one thread per face,
// both split parts), then k_ls_stage forms L(phi) per cell in the
// reference's order and applies the stage.  All arithmetic is FP64 with every
// product rounded on its own (a fused multiply-add only where one factor is a
// power of two, which rounds the same), so the results equal the FP64 oracle
// bit for bit.  GB300's FP64 pipe runs at about 1/57 of its FP32 rate and
// these kernels are bound by it, not by memory; what is kept off it:
//   - every division and most multiplications: correctly rounded quotients and
//     products in integer and FP32 arithmetic (idiv.h), one reciprocal per
//     divisor;
//   - what neighbouring faces share: the smoothness indicators and weights of
//     a three-cell stencil are formed once per cell and handed along the line
//     through shared memory, where they were formed once per face and side;
//   - the side the flow does not come from: a split flux that is zero on a
//     stencil has constant weights, and a face value of zeros is a zero.
// Measured: a 256^3 advection step with a smooth velocity 92.8 -> 17.7 ms (with
// the divisions alone off the pipe 22.9), one redistancing call of 13
// iterations on 143x127x101 cells 139.0 -> 28.7 ms (37.1).  The face kernel
// issues 46 FP64 warp instructions per 32 cells of a 128^3 case (about 355
// before) and runs at 59% of the FP64 pipe and 46% of the issue slots: the
// integer work that replaced the rest now takes about as long.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>

#include "gbmg.h"
#include "gbmg_internal.h"
#include "idiv.h"

namespace gbmg {

namespace {

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dvd(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ double by3(double a) { return div_3(a, 0); }
__device__ __forceinline__ double by6(double a) { return div_3(a, 1); }
__device__ __forceinline__ double by12(double a) { return div_3(a, 2); }
__device__ __forceinline__ double by4(double a) { return mul(a, 0.25); }  // exact
// a + c b with c b exact (c a power of two): the sum's one rounding
__device__ __forceinline__ double fma2(double c, double b, double a) { return __fma_rn(c, b, a); }

__device__ __forceinline__ double isq(double x) { return mul_int(x, x); }

// eps + b1, eps + b2, eps + b3 squared for the three-cell stencil (ga, gb, gc):
// the indicators of a left-biased face two cells to the right of ga (x[0]),
// right of gb (x[1]) and left of gc (x[2]).  ta = 3 ga, tc = 3 gc.
__device__ __forceinline__ void weno_stencil(double ga, double gb, double gc, double ta, double tc,
                                             double eps, double (&x)[3]) {
  const double d = mul_k<13>(isq(add(fma2(-2.0, gb, ga), gc)));
  x[0] = isq(add(eps, add(d, mul_k<3>(isq(add(fma2(-4.0, gb, ga), tc))))));
  x[1] = isq(add(eps, add(d, mul_k<3>(isq(sub(ga, gc))))));
  x[2] = isq(add(eps, add(d, mul_k<3>(isq(add(fma2(-4.0, gb, ta), gc))))));
}

// value at face i+1/2 of g(i-2..i+2) = g0..g4, biased to the left, from the
// unnormalised weights a1, a2, a3
__device__ __forceinline__ double weno_left(double a1, double a2, double a3, double g0, double g1,
                                            double g2, double g3, double g4) {
  const RcpInt s = rcp_int(add(add(a1, a2), a3));
  const double w1 = div_int(a1, s), w2 = div_int(a2, s), w3 = div_int(a3, s);
  double v = mul_int(by3(w1), g0);
  v = sub(v, mul_int(by6(add(mul_k<7>(w1), w2)), g1));
  v = add(v, mul_int(by6(fma2(2.0, w3, add(mul_k<11>(w1), mul_k<5>(w2)))), g2));
  v = add(v, mul_int(by6(fma2(2.0, w2, mul_k<5>(w3))), g3));
  v = sub(v, mul_int(by6(w3), g4));
  return v;
}

// value at face i+1/2 of f(i-1..i+3) = f0..f4, biased to the right
__device__ __forceinline__ double weno_right(double a1, double a2, double a3, double f0, double f1,
                                             double f2, double f3, double f4) {
  const RcpInt s = rcp_int(add(add(a1, a2), a3));
  const double w1 = div_int(a1, s), w2 = div_int(a2, s), w3 = div_int(a3, s);
  double v = by6(mul_int(w3, fma2(2.0, f2, sub(mul_k<5>(f1), f0))));
  v = add(v, by6(mul_int(w2, sub(fma2(2.0, f1, mul_k<5>(f2)), f3))));
  v = add(v, by6(mul_int(w1, fma2(2.0, f4, sub(mul_k<11>(f2), mul_k<7>(f3))))));
  return v;
}

__device__ __forceinline__ bool is_zero(double x) {
  return ((unsigned long long)__double_as_longlong(x) << 1) == 0ull;
}
// a zero as a float of the same sign
__device__ __forceinline__ float zero_f(double x) {
  return __int_as_float(__double2hiint(x) & (int)0x80000000);
}
__device__ __forceinline__ double zero_d(float z) {
  return __hiloint2double(__float_as_int(z), 0);
}
// weno_left and weno_right of five zeros: a zero, its sign from the same sums
__device__ __forceinline__ double weno_left_zero(double g0, double g1, double g2, double g3,
                                                 double g4) {
  return zero_d(__fsub_rn(
      __fadd_rn(__fadd_rn(__fsub_rn(zero_f(g0), zero_f(g1)), zero_f(g2)), zero_f(g3)), zero_f(g4)));
}
__device__ __forceinline__ double weno_right_zero(double d0, double d1, double d2, double d3,
                                                  double d4) {
  const float f0 = zero_f(d0), f1 = zero_f(d1), f2 = zero_f(d2), f3 = zero_f(d3), f4 = zero_f(d4);
  float v = __fadd_rn(__fadd_rn(-f0, f1), f2);
  v = __fadd_rn(v, __fsub_rn(__fadd_rn(f1, f2), f3));
  return zero_d(__fadd_rn(v, __fadd_rn(__fsub_rn(f2, f3), f4)));
}

__device__ __forceinline__ int clampi(int i, int n) { return i < 0 ? 0 : (i >= n ? n - 1 : i); }

struct LsGrid {
  int nx, ny, nz;
  ConstDiv h[3];
};

LsGrid ls_grid(const gbmg_grid& g) {
  return LsGrid{g.nx, g.ny, g.nz, {const_div(g.dx), const_div(g.dy), const_div(g.dz)}};
}

// A block works on kLines lines of kSeg consecutive cells along an axis, one
// thread per cell; what a cell's face needs of its neighbours goes through
// shared memory.  The face right of a cell needs three-cell stencils up to two
// cells away, so kFaces = kSeg - 5 faces of a segment are complete.  A warp is
// 8 lines by 4 cells for every axis: the lines are adjacent along x (64-byte
// accesses), or along y for the x axis (32-byte accesses), where it keeps the
// ends of segments from idling half a warp (the kernels are bound by
// arithmetic, with DRAM at a few percent).
constexpr int kSeg = 64, kLines = 8, kLsThreads = kSeg * kLines, kFaces = kSeg - 5;

struct LsLine {
  int c;         // the thread's cell along the axis (may lie outside the grid)
  int a;         // position in the segment
  int n;         // cells along the axis
  int l1, l2;    // the line: its two other indices
  bool live;     // the line exists
  size_t stride, base;
};

// The unit of a block: count = (segments) x (line groups) x (other axis)
template <int kAxis>
__device__ __forceinline__ LsLine ls_line(const LsGrid& g, int faces) {
  LsLine L;
  L.a = threadIdx.x / kLines;
  const int l = threadIdx.x % kLines;
  L.n = kAxis == 0 ? g.nx : (kAxis == 1 ? g.ny : g.nz);
  const int n1 = kAxis == 0 ? g.ny : g.nx;
  const int segs = (faces + kFaces - 1) / kFaces, groups = (n1 + kLines - 1) / kLines;
  const unsigned b = blockIdx.x;
  const int seg = (int)(b % (unsigned)segs);
  const unsigned r = b / (unsigned)segs;
  L.l1 = (int)(r % (unsigned)groups) * kLines + l;
  L.l2 = (int)(r / (unsigned)groups);
  L.live = L.l1 < n1;
  const int l1 = L.live ? L.l1 : n1 - 1;
  L.c = seg * kFaces - 3 + L.a;
  L.stride = kAxis == 0 ? 1 : (kAxis == 1 ? (size_t)g.nx : (size_t)g.nx * g.ny);
  L.base = kAxis == 0   ? ((size_t)L.l2 * g.ny + l1) * g.nx
           : kAxis == 1 ? (size_t)L.l2 * g.ny * g.nx + l1
                        : (size_t)L.l2 * g.nx + l1;
  return L;
}

unsigned ls_blocks(const LsGrid& g, int axis, int faces) {
  const int n1 = axis == 0 ? g.ny : g.nx, n2 = axis == 2 ? g.ny : g.nz;
  return (unsigned)((faces + kFaces - 1) / kFaces) * (unsigned)((n1 + kLines - 1) / kLines) *
         (unsigned)n2;
}

// weights of a stencil of zeros: 1, 6 and 3 over eps^2
struct LsZero {
  double w1, w6, w3;
};

LsZero ls_zero(double eps) {
  const double x = eps * eps;
  return LsZero{1.0 / x, 6.0 / x, 3.0 / x};
}

constexpr double kAdvEps = 1.0e-13, kRedisEps = 1.0e-10;

// Faces of one axis: face f (0..n) is the reference's face i+1/2 with
// i = f - 1; ss1 = left-biased WENO of u+ phi, ss2 = right-biased of u- phi.
// The face arrays are laid out like cell arrays with n+1 entries along the
// axis.
template <int kAxis>
__global__ void __launch_bounds__(kLsThreads, 2)
    k_ls_faces(LsGrid g, LsZero z, const double* __restrict__ phi, const double* __restrict__ vel,
               double* __restrict__ ss1, double* __restrict__ ss2) {
  constexpr int S = kLines;  // neighbour along the line
  __shared__ double gp[kLsThreads], gm[kLsThreads], tp[kLsThreads], tm[kLsThreads];
  __shared__ double p1[kLsThreads], p3[kLsThreads], m1[kLsThreads], m2[kLsThreads];
  const int t = threadIdx.x;
  const LsLine L = ls_line<kAxis>(g, (kAxis == 0 ? g.nx : kAxis == 1 ? g.ny : g.nz) + 1);
  const bool used = L.live && L.c <= L.n + 2;  // cells that some face reads
  if (used) {
    const size_t q = L.base + (size_t)clampi(L.c, L.n) * L.stride;
    const double u = vel[q], p = phi[q];
    double a, b;
    const long long ub = __double_as_longlong(u);
    if ((ub & 0x7ff0000000000000ll) < 0x7fe0000000000000ll &&
        (__double_as_longlong(p) & 0x7ff0000000000000ll) < 0x7ff0000000000000ll) {
      // (u + |u|)/2 and (u - |u|)/2 are u and +0, or +0 and u (-0 keeps its
      // sign in the second): one product, the other a zero of p's sign
      const double v = mul_int(u, p);
      const double zp = __hiloint2double(__double2hiint(p) & (int)0x80000000, 0);
      const bool neg = ub < 0, nz = (ub << 1) != 0;
      a = !neg && nz ? v : zp;
      b = neg ? v : zp;
    } else {
      a = mul(mul(0.5, add(u, fabs(u))), p);
      b = mul(mul(0.5, sub(u, fabs(u))), p);
    }
    gp[t] = a;
    gm[t] = b;
    tp[t] = mul_k<3>(a);
    tm[t] = mul_k<3>(b);
  }
  __syncthreads();
  double p2 = z.w6, m3 = z.w3;
  if (used && L.a >= 1 && L.a <= kSeg - 2 && L.c <= L.n + 1) {
    double x[3], w1 = z.w1, w3 = z.w3;
    if (!(is_zero(gp[t - S]) && is_zero(gp[t]) && is_zero(gp[t + S]))) {
      weno_stencil(gp[t - S], gp[t], gp[t + S], tp[t - S], tp[t + S], kAdvEps, x);
      w1 = div_int(1.0, rcp_int(x[0]));
      p2 = div_int(6.0, rcp_int(x[1]));
      w3 = div_int(3.0, rcp_int(x[2]));
    }
    p1[t] = w1;
    p3[t] = w3;
    w1 = z.w1;
    double w2 = z.w6;
    if (!(is_zero(gm[t - S]) && is_zero(gm[t]) && is_zero(gm[t + S]))) {
      weno_stencil(gm[t - S], gm[t], gm[t + S], tm[t - S], tm[t + S], kAdvEps, x);
      w1 = div_int(1.0, rcp_int(x[2]));
      w2 = div_int(6.0, rcp_int(x[1]));
      m3 = div_int(3.0, rcp_int(x[0]));
    }
    m1[t] = w1;
    m2[t] = w2;
  }
  __syncthreads();
  const int f = L.c + 1;
  if (!L.live || L.a < 2 || L.a > kSeg - 4 || f > L.n) return;
  const int ex = g.nx + (kAxis == 0), ey = g.ny + (kAxis == 1);
  const size_t o = kAxis == 0   ? ((size_t)L.l2 * ey + L.l1) * ex + f
                   : kAxis == 1 ? ((size_t)L.l2 * ey + f) * ex + L.l1
                                : ((size_t)f * ey + L.l2) * ex + L.l1;
  {
    const double g0 = gp[t - 2 * S], g1 = gp[t - S], g2 = gp[t], g3 = gp[t + S], g4 = gp[t + 2 * S];
    if (is_zero(g0) && is_zero(g1) && is_zero(g2) && is_zero(g3) && is_zero(g4))
      ss1[o] = weno_left_zero(g0, g1, g2, g3, g4);
    else
      ss1[o] = weno_left(p1[t - S], p2, p3[t + S], g0, g1, g2, g3, g4);
  }
  {
    const double f0 = gm[t - S], f1 = gm[t], f2 = gm[t + S], f3 = gm[t + 2 * S], f4 = gm[t + 3 * S];
    if (is_zero(f0) && is_zero(f1) && is_zero(f2) && is_zero(f3) && is_zero(f4))
      ss2[o] = weno_right_zero(f0, f1, f2, f3, f4);
    else
      ss2[o] = weno_right(m1[t + 2 * S], m2[t + S], m3, f0, f1, f2, f3, f4);
  }
}

// One stage: l = L(phi) per cell, then phi += src * dt with the stage's
// combination of l1, l2, l3 (level_set_rk3_solver).
__global__ void __launch_bounds__(256) k_ls_stage(LsGrid g, int stage, double dt,
                                                  const double* __restrict__ x1,
                                                  const double* __restrict__ x2,
                                                  const double* __restrict__ y1,
                                                  const double* __restrict__ y2,
                                                  const double* __restrict__ z1,
                                                  const double* __restrict__ z2, double* l1,
                                                  double* l2, double* phi) {
  const size_t n = (size_t)g.nx * g.ny * g.nz;
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const int i = (int)(q % g.nx);
  const size_t r = q / g.nx;
  const int j = (int)(r % g.ny), k = (int)(r / g.ny);
  // face indices: high face of the cell = low face + one step along the axis
  const size_t fx = ((size_t)k * g.ny + j) * (g.nx + 1) + i;
  const size_t fy = ((size_t)k * (g.ny + 1) + j) * g.nx + i;
  const size_t fz = ((size_t)k * g.ny + j) * g.nx + i;
  double d = sub(sub(add(x1[fx + 1], x2[fx + 1]), x1[fx]), x2[fx]);
  double src = -div_const(g.h[0], d);
  d = sub(sub(add(y1[fy + g.nx], y2[fy + g.nx]), y1[fy]), y2[fy]);
  src = sub(src, div_const(g.h[1], d));
  if (g.nz > 1) {
    const size_t pz = (size_t)g.nx * g.ny;
    d = sub(sub(add(z1[fz + pz], z2[fz + pz]), z1[fz]), z2[fz]);
    src = sub(src, div_const(g.h[2], d));
  }
  double s;
  if (stage == 1) {
    l1[q] = src;
    s = src;
  } else if (stage == 2) {
    l2[q] = src;
    s = by4(sub(src, mul_k<3>(l1[q])));
  } else {
    s = by12(fma2(8.0, src, sub(-l1[q], l2[q])));
  }
  phi[q] = add(phi[q], mul_int(s, dt));
}

// ---- redistancing: level_set_rk3_redis ("Two phase flows/newOpenMP/2D/src/
// interface_solver/level_set_rk3_redis.f90:1-361"; 3D "Two phase flows/
// newOpenMP/3D+IBM/src/interface_solver/level_set_rk3_redis.f90") ----------
constexpr double kPi = 3.141592653589793;  // acos(-1) in double

// ls_funs ("Two phase flows/newOpenMP/3D+IBM/src/interface_solver/
// others.f90:1-37"): smoothed Heaviside, its derivative and the sign 2H - 1.
// Beyond `out` (slightly above ls_wid (1 - 1e-12), from the host) phi/ls_wid
// lands past the clipping threshold, so H is 0 or 1 without the division; the
// test compares bit patterns (NaN takes the formula).
struct LsWidth {
  double wid;
  long long out;
};

LsWidth ls_width(double ls_wid) {
  return LsWidth{ls_wid, ls_outside_bits(ls_wid)};
}

__device__ __forceinline__ bool ls_outside(const LsWidth& w, double phi) {
  const long long m = __double_as_longlong(phi) & 0x7fffffffffffffffll;
  return m > w.out && m <= 0x7ff0000000000000ll;
}

__device__ __forceinline__ void ls_funs1(double phi, const LsWidth& w, double& heavy,
                                         double& delta, double& sgn) {
  if (ls_outside(w, phi)) {
    const bool neg = __double_as_longlong(phi) < 0;
    heavy = neg ? 0.0 : 1.0;
    delta = 0.0;
    sgn = neg ? -1.0 : 1.0;
    return;
  }
  const double eps = 1.0e-12;
  const double x = dvd(phi, w.wid);
  double h, hp;
  if (x > 1.0 - eps) {
    h = 1.0;
    hp = 0.0;
  } else if (x < -1.0 + eps) {
    h = 0.0;
    hp = 0.0;
  } else {
    h = mul(0.5, add(add(1.0, x), dvd(sin(mul(kPi, x)), kPi)));
    hp = dvd(mul(0.5, add(1.0, cos(mul(kPi, x)))), w.wid);
  }
  h = h < 1.0 ? h : 1.0;
  h = h > 0.0 ? h : 0.0;
  heavy = h;
  delta = hp;
  sgn = sub(mul(2.0, h), 1.0);
}

// s = the sign held fixed through the call: 2H - 1, or phi itself for the
// first redistancing (level_set_redis_stable, btn = 0)
__global__ void __launch_bounds__(256) k_ls_sign(size_t n, const double* __restrict__ phi,
                                                 LsWidth ls_wid, int btn,
                                                 double* __restrict__ s) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  if (btn == 0) {
    s[q] = phi[q];
  } else {
    double hv, dl, sg;
    ls_funs1(phi[q], ls_wid, hv, dl, sg);
    s[q] = sg;
  }
}

__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }

// max(x, 0) and max(-x, 0), 0 for NaN, and the larger of two such values, by
// their bit patterns (FP64 comparisons run on the FP64 pipe)
__device__ __forceinline__ double pos_part(double x) {
  const long long b = __double_as_longlong(x);
  return b > 0 && b <= 0x7ff0000000000000ll ? x : 0.0;
}
__device__ __forceinline__ double neg_part(double x) {
  return pos_part(__hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x)));
}
__device__ __forceinline__ double larger(double a, double b) {
  return __double_as_longlong(a) > __double_as_longlong(b) ? a : b;
}
__device__ __forceinline__ bool at_least_zero(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return b <= 0x7ff0000000000000ull || b == 0x8000000000000000ull;
}

// |grad phi| by Godunov upwinding on the sign s (level_set_redis_gradient):
// the WENO-JS one-sided values (EPS = 1e-10) of the backward differences
// (phi_i - phi_{i-1})/h, zero-gradient ghosts by index clamping.  One launch
// per axis, which adds its square to grad; both sides' weights of a stencil
// come from the same three indicators.  The last axis takes the root and, with
// kLambda, forms s2 = lam s (|grad| - 1) and s3 = |grad| delta lam
// (level_set_redis_lambda; delta and both are 0 outside the band) and raises
// *odd when one of them is not finite.
template <int kAxis, bool kLast, bool kLambda>
__global__ void __launch_bounds__(kLsThreads, 2)
    k_ls_grad(LsGrid g, const double* __restrict__ phi, const double* __restrict__ s,
              double* __restrict__ grad, LsWidth wid, double rho12, double* __restrict__ s2,
              double* __restrict__ s3, unsigned long long* odd) {
  constexpr int S = kLines;
  __shared__ double d[kLsThreads], td[kLsThreads];
  __shared__ double l1[kLsThreads], l3[kLsThreads], r1[kLsThreads], r2[kLsThreads];
  const int t = threadIdx.x;
  const LsLine L = ls_line<kAxis>(g, (kAxis == 0 ? g.nx : kAxis == 1 ? g.ny : g.nz) + 1);
  const bool used = L.live && L.c <= L.n + 2;
  if (used) {
    const int cc = clampi(L.c, L.n), cm = cc > 0 ? cc - 1 : 0;
    const double v = div_const(g.h[kAxis], sub(phi[L.base + (size_t)cc * L.stride],
                                               phi[L.base + (size_t)cm * L.stride]));
    d[t] = v;
    td[t] = mul_k<3>(v);
  }
  __syncthreads();
  double w2 = 0.0, w3 = 0.0;
  if (used && L.a >= 1 && L.a <= kSeg - 2 && L.c <= L.n + 1) {
    double x[3];
    weno_stencil(d[t - S], d[t], d[t + S], td[t - S], td[t + S], kRedisEps, x);
    const RcpInt x0 = rcp_int(x[0]);
    l1[t] = div_int(1.0, x0);
    w3 = div_int(3.0, x0);
    w2 = div_int(6.0, rcp_int(x[1]));
    r2[t] = w2;
    const RcpInt x2 = rcp_int(x[2]);
    r1[t] = div_int(1.0, x2);
    l3[t] = div_int(3.0, x2);
  }
  __syncthreads();
  if (!L.live || L.a < 2 || L.a > kSeg - 4 || L.c < 0 || L.c >= L.n) return;
  const size_t q = L.base + (size_t)L.c * L.stride;
  const double sq = s[q];
  const double v1 = weno_right(r1[t + 2 * S], r2[t + S], w3, d[t - S], d[t], d[t + S], d[t + 2 * S],
                               d[t + 3 * S]);
  const double v2 = weno_left(l1[t - S], w2, l3[t + S], d[t - 2 * S], d[t - S], d[t], d[t + S],
                              d[t + 2 * S]);
  const double v = at_least_zero(sq) ? larger(neg_part(v1), pos_part(v2))
                                     : larger(pos_part(v1), neg_part(v2));
  double sum = isq(v);
  if (kAxis > 0) sum = add(grad[q], sum);
  if (kLast) sum = sqrt_int(sum);
  grad[q] = sum;
  if (kLast && kLambda) {
    const double p = phi[q];
    double a = 0.0, b = 0.0;
    if (!ls_outside(wid, p) ||
        (__double_as_longlong(sum) & 0x7ff0000000000000ll) == 0x7ff0000000000000ll) {
      double hv, dl, sg;
      ls_funs1(p, wid, hv, dl, sg);
      const double lam = g.nz > 1 ? mul(add(mul(mul(2.0, sub(1.0, rho12)), hv), rho12), dl) : dl;
      a = mul(mul(lam, sq), sub(sum, 1.0));
      b = mul(mul(sum, dl), lam);
      const long long e = 0x7ff0000000000000ll;
      if ((__double_as_longlong(a) & e) == e || (__double_as_longlong(b) & e) == e)
        atomicOr(odd, 1ull);
    }
    s2[q] = a;
    s3[q] = b;
  }
}

// One pseudo-time stage: s1 = the correction (block sums of s2 and s3 with
// weight 16 (2D) or 51 (3D) on the cell, btn = 1; 0 for btn = 0),
// l = (s - s1)|grad| - s, phi -= rdt * (the stage's combination of l1..l3).
// s1 carries the factor delta, so it is 0 outside the band and only the
// band's cells add the 54 neighbours (unless one of s2, s3 is not finite
// somewhere, *odd).
__global__ void __launch_bounds__(256) k_ls_redis_stage(LsGrid g, int stage, int btn, double rdt,
                                                        LsWidth ls_wid,
                                                        const unsigned long long* odd,
                                                        const double* __restrict__ s,
                                                        const double* __restrict__ grad,
                                                        const double* __restrict__ s2,
                                                        const double* __restrict__ s3,
                                                        double* l1, double* l2, double* phi) {
  const size_t n = (size_t)g.nx * g.ny * g.nz;
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  double s1 = 0.0;
  if (btn != 0 && (!ls_outside(ls_wid, phi[q]) || *odd != 0ull)) {
    const int i = (int)(q % g.nx);
    const size_t r = q / g.nx;
    const int j = (int)(r % g.ny), k = (int)(r / g.ny);
    const bool three = g.nz > 1;
    const double wgt = three ? 51.0 : 16.0;
    double a = mul(wgt, s2[q]), b = mul(wgt, s3[q]);
    const int k0 = three ? -1 : 0, k1 = three ? 1 : 0;
    for (int kk = k0; kk <= k1; ++kk)
      for (int jj = -1; jj <= 1; ++jj)
        for (int ii = -1; ii <= 1; ++ii) {
          const size_t rr = ((size_t)clampi(k + kk, g.nz) * g.ny + clampi(j + jj, g.ny)) * g.nx +
                            clampi(i + ii, g.nx);
          a = add(a, s2[rr]);
          b = add(b, s3[rr]);
        }
    double hv, dl, sg;
    ls_funs1(phi[q], ls_wid, hv, dl, sg);
    s1 = fabs(b) > 1.0e-12 ? mul(dvd(a, b), dl) : 0.0;
  }
  const double l = sub(mul_int(sub(s[q], s1), grad[q]), s[q]);
  double src;
  if (stage == 1) {
    l1[q] = l;
    src = l;
  } else if (stage == 2) {
    l2[q] = l;
    src = by4(sub(l, mul_k<3>(l1[q])));
  } else {
    src = by12(fma2(8.0, l, sub(-l1[q], l2[q])));
  }
  phi[q] = sub(phi[q], mul_int(rdt, src));
}

// *out = max over cells of |a - b| (b == nullptr: max of a, a >= 0); the
// maximum of non-negative doubles is the maximum of their bit patterns
__global__ void __launch_bounds__(256) k_ls_maxabs(size_t n, const double* __restrict__ a,
                                                   const double* __restrict__ b,
                                                   unsigned long long* out) {
  double m = 0.0;
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n;
       q += (size_t)gridDim.x * blockDim.x) {
    const double v = b ? fabs(sub(a[q], b[q])) : a[q];
    m = v > m ? v : m;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = dmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double ws[8];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = dmax(m, ws[w]);
    atomicMax(out, (unsigned long long)__double_as_longlong(m));
  }
}

__global__ void k_ls_scale(size_t n, double* phi, const unsigned long long* gmax) {
  const double gm = __longlong_as_double((long long)*gmax);
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) phi[q] = dvd(phi[q], gm);
}

inline unsigned blocks_for(size_t n) { return (unsigned)((n + 255) / 256); }

}  // namespace

}  // namespace gbmg

using namespace gbmg;

struct gbmg_ls {
  gbmg_grid grid{};
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  double *phi = nullptr, *u = nullptr, *v = nullptr, *w = nullptr, *l1 = nullptr, *l2 = nullptr;
  double* face[6] = {};
  unsigned long long* red = nullptr;  // a max-reduction slot and a flag
  unsigned long long* host_red = nullptr;
  int64_t launches = 0;
  std::string err;
};

namespace {

int ls_fail(gbmg_ls* ls, cudaError_t e, const char* what) {
  ls->err = std::string(what) + ": " + cudaGetErrorString(e);
  return e == cudaErrorMemoryAllocation ? GBMG_OUT_OF_MEMORY : GBMG_CUDA_ERROR;
}

#define LS_CUDA(ls, call)                              \
  do {                                                 \
    cudaError_t e_ = (call);                           \
    if (e_ != cudaSuccess) return ls_fail(ls, e_, #call); \
  } while (0)

size_t ls_cells(const gbmg_grid& g) { return (size_t)g.nx * g.ny * g.nz; }

void ls_free(gbmg_ls* ls) {
  double** all[] = {&ls->phi, &ls->u, &ls->v, &ls->w, &ls->l1, &ls->l2, &ls->face[0], &ls->face[1],
                    &ls->face[2], &ls->face[3], &ls->face[4], &ls->face[5]};
  for (double** p : all)
    if (*p) {
      cudaFree(*p);
      *p = nullptr;
    }
  if (ls->red) cudaFree(ls->red);
  if (ls->host_red) cudaFreeHost(ls->host_red);
  ls->red = nullptr;
  ls->host_red = nullptr;
}

// host or device field (strided, x contiguous) -> dense device array
int ls_in(gbmg_ls* ls, const gbmg_field& f, int mem, double* dst) {
  const gbmg_grid& g = ls->grid;
  if (!f.data || f.sy < g.nx || f.sz < f.sy * (int64_t)g.ny) {
    ls->err = "invalid field";
    return GBMG_INVALID_ARG;
  }
  const bool dense = f.sy == g.nx && f.sz == (int64_t)g.nx * g.ny;
  if (dense) {
    LS_CUDA(ls, cudaMemcpyAsync(dst, f.data, ls_cells(g) * sizeof(double),
                                mem == GBMG_MEM_HOST ? cudaMemcpyHostToDevice
                                                     : cudaMemcpyDeviceToDevice,
                                ls->stream));
  } else if (mem == GBMG_MEM_DEVICE) {
    launch_copy_in(ls->stream, g.nx, g.ny, g.nz, Strided{f.data, f.sy, f.sz}, dst);
    ls->launches += 1;
    LS_CUDA(ls, cudaGetLastError());
  } else {
    for (int k = 0; k < g.nz; ++k)
      LS_CUDA(ls, cudaMemcpy2DAsync(dst + (size_t)k * g.nx * g.ny, (size_t)g.nx * sizeof(double),
                                    f.data + (int64_t)k * f.sz, (size_t)f.sy * sizeof(double),
                                    (size_t)g.nx * sizeof(double), (size_t)g.ny,
                                    cudaMemcpyHostToDevice, ls->stream));
  }
  return GBMG_OK;
}

int ls_out(gbmg_ls* ls, const double* src, int mem, const gbmg_field& f) {
  const gbmg_grid& g = ls->grid;
  const bool dense = f.sy == g.nx && f.sz == (int64_t)g.nx * g.ny;
  if (dense) {
    LS_CUDA(ls, cudaMemcpyAsync(f.data, src, ls_cells(g) * sizeof(double),
                                mem == GBMG_MEM_HOST ? cudaMemcpyDeviceToHost
                                                     : cudaMemcpyDeviceToDevice,
                                ls->stream));
  } else if (mem == GBMG_MEM_DEVICE) {
    launch_copy_out(ls->stream, g.nx, g.ny, g.nz, src, f.data, f.sy, f.sz);
    ls->launches += 1;
    LS_CUDA(ls, cudaGetLastError());
  } else {
    for (int k = 0; k < g.nz; ++k)
      LS_CUDA(ls, cudaMemcpy2DAsync(f.data + (int64_t)k * f.sz, (size_t)f.sy * sizeof(double),
                                    src + (size_t)k * g.nx * g.ny, (size_t)g.nx * sizeof(double),
                                    (size_t)g.nx * sizeof(double), (size_t)g.ny,
                                    cudaMemcpyDeviceToHost, ls->stream));
  }
  return GBMG_OK;
}

}  // namespace

extern "C" {

int gbmg_ls_create(const gbmg_grid* grid, int device, void* stream, gbmg_ls** out) {
  if (!grid || !out) return GBMG_INVALID_ARG;
  *out = nullptr;
  if (grid->nx < 1 || grid->ny < 1 || grid->nz < 1 || !(grid->dx > 0) || !(grid->dy > 0) ||
      (grid->nz > 1 && !(grid->dz > 0)))
    return GBMG_INVALID_ARG;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return GBMG_NO_DEVICE;
  gbmg_ls* ls = new gbmg_ls();
  ls->grid = *grid;
  if (device < 0) cudaGetDevice(&device);
  ls->device = device;
  if (cudaSetDevice(device) != cudaSuccess) {
    delete ls;
    return GBMG_NO_DEVICE;
  }
  if (stream) {
    ls->stream = static_cast<cudaStream_t>(stream);
  } else {
    if (cudaStreamCreateWithFlags(&ls->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete ls;
      return GBMG_CUDA_ERROR;
    }
    ls->own_stream = true;
  }
  const gbmg_grid& g = *grid;
  const size_t n = ls_cells(g);
  const size_t nfx = (size_t)(g.nx + 1) * g.ny * g.nz, nfy = (size_t)g.nx * (g.ny + 1) * g.nz,
               nfz = (size_t)g.nx * g.ny * (g.nz + 1);
  const size_t sizes[12] = {n, n, n, n, n, n, nfx, nfx, nfy, nfy, nfz, nfz};
  double** ptrs[12] = {&ls->phi, &ls->u, &ls->v, &ls->w, &ls->l1, &ls->l2, &ls->face[0],
                       &ls->face[1], &ls->face[2], &ls->face[3], &ls->face[4], &ls->face[5]};
  for (int a = 0; a < 12; ++a) {
    if (cudaMalloc((void**)ptrs[a], sizes[a] * sizeof(double)) != cudaSuccess) {
      cudaGetLastError();
      ls_free(ls);
      if (ls->own_stream) cudaStreamDestroy(ls->stream);
      delete ls;
      return GBMG_OUT_OF_MEMORY;
    }
  }
  if (cudaMalloc((void**)&ls->red, 2 * sizeof(unsigned long long)) != cudaSuccess ||
      cudaMallocHost((void**)&ls->host_red, sizeof(unsigned long long)) != cudaSuccess) {
    cudaGetLastError();
    ls_free(ls);
    if (ls->own_stream) cudaStreamDestroy(ls->stream);
    delete ls;
    return GBMG_OUT_OF_MEMORY;
  }
  *out = ls;
  return GBMG_OK;
}

int gbmg_ls_destroy(gbmg_ls* ls) {
  if (!ls) return GBMG_INVALID_ARG;
  cudaSetDevice(ls->device);
  if (ls->stream) cudaStreamSynchronize(ls->stream);
  ls_free(ls);
  if (ls->own_stream && ls->stream) cudaStreamDestroy(ls->stream);
  delete ls;
  return GBMG_OK;
}

int gbmg_ls_advect(gbmg_ls* ls, gbmg_field phi, gbmg_field u, gbmg_field v, gbmg_field w,
                   double dt, int steps, int mem) {
  if (!ls) return GBMG_INVALID_ARG;
  ls->err.clear();
  if (cudaSetDevice(ls->device) != cudaSuccess) {
    ls->err = "cudaSetDevice failed";
    return GBMG_CUDA_ERROR;
  }
  if (!(dt > 0) || steps < 0) {
    ls->err = "dt must be > 0 and steps >= 0";
    return GBMG_INVALID_ARG;
  }
  if (mem != GBMG_MEM_HOST && mem != GBMG_MEM_DEVICE) {
    ls->err = "mem must be GBMG_MEM_HOST or GBMG_MEM_DEVICE";
    return GBMG_INVALID_ARG;
  }
  const gbmg_grid& g = ls->grid;
  const bool three = g.nz > 1;
  int rc;
  if ((rc = ls_in(ls, phi, mem, ls->phi)) != GBMG_OK) return rc;
  if ((rc = ls_in(ls, u, mem, ls->u)) != GBMG_OK) return rc;
  if ((rc = ls_in(ls, v, mem, ls->v)) != GBMG_OK) return rc;
  if (three && (rc = ls_in(ls, w, mem, ls->w)) != GBMG_OK) return rc;
  const LsGrid G = ls_grid(g);
  const size_t n = ls_cells(g);
  const double* vel[3] = {ls->u, ls->v, ls->w};
  const LsZero Z = ls_zero(kAdvEps);
  for (int s = 0; s < steps; ++s)
    for (int stage = 1; stage <= 3; ++stage) {
      k_ls_faces<0><<<ls_blocks(G, 0, g.nx + 1), kLsThreads, 0, ls->stream>>>(
          G, Z, ls->phi, vel[0], ls->face[0], ls->face[1]);
      k_ls_faces<1><<<ls_blocks(G, 1, g.ny + 1), kLsThreads, 0, ls->stream>>>(
          G, Z, ls->phi, vel[1], ls->face[2], ls->face[3]);
      if (three)
        k_ls_faces<2><<<ls_blocks(G, 2, g.nz + 1), kLsThreads, 0, ls->stream>>>(
            G, Z, ls->phi, vel[2], ls->face[4], ls->face[5]);
      ls->launches += three ? 3 : 2;
      k_ls_stage<<<blocks_for(n), 256, 0, ls->stream>>>(
          G, stage, dt, ls->face[0], ls->face[1], ls->face[2], ls->face[3], ls->face[4],
          ls->face[5], ls->l1, ls->l2, ls->phi);
      ls->launches += 1;
    }
  LS_CUDA(ls, cudaGetLastError());
  if ((rc = ls_out(ls, ls->phi, mem, phi)) != GBMG_OK) return rc;
  LS_CUDA(ls, cudaStreamSynchronize(ls->stream));
  return GBMG_OK;
}

namespace {
// |grad phi| of ls->phi, one launch per axis; with lambda also s2 and s3
void ls_gradient(gbmg_ls* ls, const LsGrid& G, const double* s, double* grad, bool lambda,
                 const LsWidth& wid, double rho_12, double* s2, double* s3) {
  const bool three = G.nz > 1;
  unsigned long long* odd = ls->red + 1;
  const unsigned b0 = ls_blocks(G, 0, G.nx + 1), b1 = ls_blocks(G, 1, G.ny + 1);
  const cudaStream_t st = ls->stream;
  const double* p = ls->phi;
  k_ls_grad<0, false, false><<<b0, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
  if (three) {
    const unsigned b2 = ls_blocks(G, 2, G.nz + 1);
    k_ls_grad<1, false, false><<<b1, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
    if (lambda)
      k_ls_grad<2, true, true><<<b2, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
    else
      k_ls_grad<2, true, false><<<b2, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
  } else if (lambda) {
    k_ls_grad<1, true, true><<<b1, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
  } else {
    k_ls_grad<1, true, false><<<b1, kLsThreads, 0, st>>>(G, p, s, grad, wid, rho_12, s2, s3, odd);
  }
  ls->launches += three ? 3 : 2;
}

// max over cells of |a - b| (or of a), read back to the host
int ls_max(gbmg_ls* ls, const double* a, const double* b, double* out) {
  const size_t n = ls_cells(ls->grid);
  LS_CUDA(ls, cudaMemsetAsync(ls->red, 0, sizeof(unsigned long long), ls->stream));
  unsigned blocks = blocks_for(n);
  if (blocks > 1024) blocks = 1024;
  k_ls_maxabs<<<blocks, 256, 0, ls->stream>>>(n, a, b, ls->red);
  ls->launches += 1;
  LS_CUDA(ls, cudaGetLastError());
  LS_CUDA(ls, cudaMemcpyAsync(ls->host_red, ls->red, sizeof(unsigned long long),
                              cudaMemcpyDeviceToHost, ls->stream));
  LS_CUDA(ls, cudaStreamSynchronize(ls->stream));
  long long bits = (long long)*ls->host_red;
  std::memcpy(out, &bits, sizeof(double));
  return GBMG_OK;
}
}  // namespace

int gbmg_ls_redistance(gbmg_ls* ls, gbmg_field phi, double ls_wid, double rdt, double rho_12,
                       int btn, int max_iter, int mem, int32_t* iters, double* last_change) {
  if (!ls) return GBMG_INVALID_ARG;
  ls->err.clear();
  if (iters) *iters = 0;
  if (last_change) *last_change = 0.0;
  if (cudaSetDevice(ls->device) != cudaSuccess) {
    ls->err = "cudaSetDevice failed";
    return GBMG_CUDA_ERROR;
  }
  if (!(ls_wid > 0) || !(rdt > 0) || max_iter < 0 || (btn != 0 && btn != 1)) {
    ls->err = "ls_wid and rdt must be > 0, max_iter >= 0, btn 0 or 1";
    return GBMG_INVALID_ARG;
  }
  if (mem != GBMG_MEM_HOST && mem != GBMG_MEM_DEVICE) {
    ls->err = "mem must be GBMG_MEM_HOST or GBMG_MEM_DEVICE";
    return GBMG_INVALID_ARG;
  }
  const gbmg_grid& g = ls->grid;
  const bool three = g.nz > 1;
  const LsGrid G = ls_grid(g);
  const size_t n = ls_cells(g);
  const unsigned nb = blocks_for(n);
  double* s = ls->face[0];
  double* grad = ls->face[1];
  double* s2 = ls->face[2];
  double* s3 = ls->face[3];
  double* tmp = ls->face[4];
  int rc;
  if ((rc = ls_in(ls, phi, mem, ls->phi)) != GBMG_OK) return rc;
  // level_set_redis_init (+ level_set_redis_stable for btn = 0)
  // (a ratio so large, or a width so small, that lam's other factors or a quotient
  // of the sums overflow makes lam * 0 a NaN: the formula decides in every cell)
  LsWidth wid = ls_width(ls_wid);
  if (std::fabs(rho_12) >= 0x1p200 || ls_wid < 0x1p-200) wid.out = 0x7fffffffffffffffll;
  LS_CUDA(ls, cudaMemsetAsync(ls->red + 1, 0, sizeof(unsigned long long), ls->stream));
  k_ls_sign<<<nb, 256, 0, ls->stream>>>(n, ls->phi, wid, btn, s);
  ls->launches += 1;
  if (btn == 0) {
    ls_gradient(ls, G, s, grad, false, wid, rho_12, s2, s3);
    LS_CUDA(ls, cudaMemsetAsync(ls->red, 0, sizeof(unsigned long long), ls->stream));
    unsigned blocks = nb > 1024 ? 1024 : nb;
    k_ls_maxabs<<<blocks, 256, 0, ls->stream>>>(n, grad, nullptr, ls->red);
    k_ls_scale<<<nb, 256, 0, ls->stream>>>(n, ls->phi, ls->red);
    ls->launches += 2;
  }
  LS_CUDA(ls, cudaGetLastError());
  const double ext = three ? std::max(std::max(g.nx * g.dx, g.ny * g.dy), g.nz * g.dz)
                           : std::max(g.nx * g.dx, g.ny * g.dy);
  const double timestop = btn == 0 ? 1.5 * ext : 3.0 * g.dx;
  const double tol = three ? 1.0e-5 : 1.0e-8;
  double time = 0.0, error = 0.0;
  int iter = 0;
  while (iter < max_iter) {
    ++iter;
    time = time + rdt;
    LS_CUDA(ls, cudaMemcpyAsync(tmp, ls->phi, n * sizeof(double), cudaMemcpyDeviceToDevice,
                                ls->stream));
    for (int stage = 1; stage <= 3; ++stage) {
      ls_gradient(ls, G, s, grad, btn != 0, wid, rho_12, s2, s3);
      k_ls_redis_stage<<<nb, 256, 0, ls->stream>>>(G, stage, btn, rdt, wid, ls->red + 1, s, grad, s2, s3,
                                                   ls->l1, ls->l2, ls->phi);
      ls->launches += 1;
    }
    LS_CUDA(ls, cudaGetLastError());
    if ((rc = ls_max(ls, tmp, ls->phi, &error)) != GBMG_OK) return rc;
    if (time > timestop || error <= tol) break;
  }
  if ((rc = ls_out(ls, ls->phi, mem, phi)) != GBMG_OK) return rc;
  LS_CUDA(ls, cudaStreamSynchronize(ls->stream));
  if (iters) *iters = iter;
  if (last_change) *last_change = error;
  return GBMG_OK;
}

int64_t gbmg_ls_kernel_launches(gbmg_ls* ls) { return ls ? ls->launches : 0; }

const char* gbmg_ls_last_error(gbmg_ls* ls) { return ls ? ls->err.c_str() : ""; }

}  // extern "C"
