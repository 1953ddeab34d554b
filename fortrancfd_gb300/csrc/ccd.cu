// Interface normals and curvature by combined compact differences (CCD) on
// sm_103a: the reference's `curv` + `surface_norms` ("Two phase flows/
// newOpenMP/2D/src/interface_solver/others_normals.f90", 3D "…/3D+IBM/…")
// with the "ccd" scheme of lib/solver/ccd_solvers.f90 and the two-by-two
// block tridiagonal solver TWIN_DEC / TWIN_BKS of lib/solver/matrix_solver.f90.
//
// Every line of the ghost-padded box along an axis (L = n + 2g points, every
// other index over its padded range) is one block tridiagonal system for
// (f', f'').  Its matrix depends only on L and h, so ccd_factor (host) factors
// it once per axis (the reference's operations in order) into a table of 16
// doubles per point that every line reads: the forward factors (row 1), the
// back-substitution factors (row 3), the diagonal blocks (row 2), the block
// determinant and its reciprocals.  k_ccd_lines runs one line per thread: the
// right-hand side (asgn_src_ccd) is formed on the fly in the forward sweep from
// a sliding window of f, and the back substitution reads the swept values
// back; the loads of a batch of points are issued a batch ahead.  Lines along
// y and z are coalesced (adjacent threads are adjacent in x); lines along x
// read with stride, served from L1.
//
// A sweep is a chain of dependent operations, so what bounds it depends on the
// number of lines.  Where they fill the GPU it is the FP64 pipe, and part of
// the work runs on the integer pipes (k_ccd_lines: 19 FP64 operations per point
// for 53); where they do not (2D) it is the chain of one warp, which
// k_ccd_lines4 shortens by giving a line four lanes.
// k_ccd_bc fills the ghost layers by zero-gradient copies (bc), k_curvature
// forms the curvature on the interior.
//
// FP64 in the reference's operand order, compiled with -fmad=false; quotients
// and products off the FP64 pipe round the same (idiv.h), so the derivatives
// equal the oracle's bit for bit.
// The curvature's (|grad phi|^2 + 1e-12)^1.5 is formed as s * sqrt(s): sqrt is
// correctly rounded, so the power is within two roundings of exact (the
// reference's pow is within about one), at a fraction of pow's FP64 cost.
#include <algorithm>
#include <cmath>

#include "gbmg_internal.h"
#include "idiv.h"
#include "reduce.cuh"

namespace gbmg {

namespace {

// f(i) of the batch of kU points from i0, clamped to the line's end
constexpr int kU = 4;
__device__ __forceinline__ void ccd_load(const double* p, int64_t st, int i0, int step, int L,
                                         double (&v)[kU]) {
#pragma unroll
  for (int u = 0; u < kU; ++u) {
    int i = i0 + u * step;
    i = i < 0 ? 0 : (i >= L ? L - 1 : i);
    v[u] = p[(int64_t)i * st];
  }
}

__device__ __forceinline__ double ccd_over(const ConstDiv& c, double x) { return div_const_i(c, x); }
// 15/16 x
__device__ __forceinline__ double ccd_1516(double x) {
  if (((unsigned)(__double2hiint(x) >> 20) & 0x7ffu) - 64u < 1900u) return scale2<-4>(mul_k<15>(x));
  return __dmul_rn(0.9375, x);
}

// x over the block determinant of a table row
__device__ __forceinline__ double ccd_det_int(const double* __restrict__ t, double x) {
  const double den = __ldg(t + 12);
  RcpInt r;
  r.b = den;
  r.y = (uint64_t)__double_as_longlong(__ldg(t + 15));
  const uint64_t u = (uint64_t)__double_as_longlong(den);
  r.m = (u & 0xfffffffffffffull) | (1ull << 52);
  r.e = r.y != 0 ? (int)(u >> 52) : 0;
  return div_int(x, r);
}

// the same in two dependent FP64 operations
__device__ __forceinline__ double ccd_det(const double* __restrict__ t, double x) {
  const double yl = __ldg(t + 14);
  if (yl != 0.0 && ((unsigned)(__double2hiint(x) >> 20) & 0x7ffu) - 123u < 1800u)
    return __fma_rn(x, __ldg(t + 13), __dmul_rn(x, yl));
  return idiv_ieee(x, __ldg(t + 12));
}

// a pass and the pointers of one of its lines: line = i1 + n1 * i2, its first
// point at i1 s1 + i2 s2 from the box origin
struct CcdLine {
  const double* f;
  double *S, *SS;
};
__device__ __forceinline__ CcdLine ccd_line(const CcdBatch& batch, const CcdArgs& c, int pass,
                                            int line) {
  const int i1 = line % c.n1, i2 = line / c.n1;
  const int64_t base = (int64_t)i1 * c.s1 + (int64_t)i2 * c.s2;
  return CcdLine{batch.f[pass] + base, batch.S[pass] + base, batch.SS[pass] + base};
}

// right-hand sides at the ends (the high end's first one negated)
__device__ __forceinline__ void ccd_end(const CcdArgs& c, double f0, double f1, double f2, double f3,
                                        double* s, double* ss) {
  *s = ccd_over(c.hd, (-3.5 * f0 + 4.0 * f1) - 0.5 * f2);
  *ss = ccd_over(c.h2d, ((34.0 / 3.0 * f0 - 83.0 / 4.0 * f1) + 10.0 * f2) - 7.0 / 12.0 * f3);
}

// Many lines: one line per thread, bound by the arithmetic pipes.  The back
// substitution keeps six of its eight products in FP64: with the forward sweep's,
// the other two and all quotients on the integer pipes the two kinds of pipe take
// about as long (curvature of 192x128x256 cells 5.43 ms before, now 2.32; 2.39 with
// all eight in FP64, 2.82 with none).  Blocks of one warp, 28 to an SM: a block
// lasts a whole line, and with 128 threads the last blocks left the SMs half idle
// (2.47 ms).
constexpr int kCcdThreads = 32;  // lines of a block

__global__ void __launch_bounds__(kCcdThreads, 28) k_ccd_lines(CcdBatch batch) {
  const int pass = blockIdx.y;
  const CcdArgs& c = batch.c[pass];
  const double* __restrict__ table = batch.table[pass];
  const int line = blockIdx.x * blockDim.x + threadIdx.x;
  if (line >= c.n1 * c.n2) return;
  const int64_t st = c.st;
  const int L = c.L;
  const CcdLine P = ccd_line(batch, c, pass, line);
  const double* __restrict__ fl = P.f;
  double* __restrict__ Sl = P.S;
  double* __restrict__ SSl = P.SS;
  // forward sweep with the right-hand side of asgn_src_ccd formed on the fly
  double fm = fl[0], fc = fl[st];
  double s, ss;
  ccd_end(c, fm, fc, fl[2 * st], fl[3 * st], &s, &ss);
  Sl[0] = s;
  SSl[0] = ss;
  double tm = mul_k<3>(fm), tc = mul_k<3>(fc);
  double nf[kU];
  ccd_load(fl, st, 2, 1, L, nf);
  for (int i0 = 1; i0 < L - 1; i0 += kU) {
    double cf[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) cf[u] = nf[u];
    ccd_load(fl, st, i0 + 1 + kU, 1, L, nf);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int i = i0 + u;
      if (i >= L - 1) break;
      const double* t = table + (size_t)i * kCcdRec;
      const double fp = cf[u], tp = mul_k<3>(fp);
      // 15/16 (f+ - f-)/h and ((3 f- - 6 f) + 3 f+)/h^2, 6 f = 2 (3 f) exactly
      double sn = ccd_over(c.hd, ccd_1516(fp - fm));
      double ssn = ccd_over(c.h2d, __fma_rn(-2.0, tc, tm) + tp);
      sn = sn - (mul_int(__ldg(t), s) + mul_int(__ldg(t + 1), ss));
      ssn = ssn - (mul_int(__ldg(t + 2), s) + mul_int(__ldg(t + 3), ss));
      s = sn;
      ss = ssn;
      Sl[(int64_t)i * st] = s;
      SSl[(int64_t)i * st] = ss;
      fm = fc;
      fc = fp;
      tm = tc;
      tc = tp;
    }
  }
  // back substitution (TWIN_BKS)
  double sol, sol2;
  {
    const int i = L - 1;
    const double* t = table + (size_t)i * kCcdRec;
    double sn, ssn;
    ccd_end(c, fl[(int64_t)i * st], fl[(int64_t)(i - 1) * st], fl[(int64_t)(i - 2) * st],
            fl[(int64_t)(i - 3) * st], &sn, &ssn);
    sn = -sn - (__ldg(t) * s + __ldg(t + 1) * ss);
    ssn = ssn - (__ldg(t + 2) * s + __ldg(t + 3) * ss);
    sol = -ccd_det_int(t, __ldg(t + 9) * ssn - __ldg(t + 11) * sn);
    sol2 = ccd_det_int(t, __ldg(t + 8) * ssn - __ldg(t + 10) * sn);
    Sl[(int64_t)i * st] = sol;
    SSl[(int64_t)i * st] = sol2;
  }
  double ns[kU], nss[kU];
  ccd_load(Sl, st, L - 2, -1, L, ns);
  ccd_load(SSl, st, L - 2, -1, L, nss);
  for (int i0 = L - 2; i0 >= 0; i0 -= kU) {
    double cs[kU], css[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      cs[u] = ns[u];
      css[u] = nss[u];
    }
    ccd_load(Sl, st, i0 - kU, -1, L, ns);
    ccd_load(SSl, st, i0 - kU, -1, L, nss);
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int i = i0 - u;
      if (i < 0) break;
      const double* t = table + (size_t)i * kCcdRec;
      const double si = cs[u] - (__dmul_rn(__ldg(t + 4), sol) + mul_int(__ldg(t + 5), sol2));
      const double ssi = css[u] - (__dmul_rn(__ldg(t + 6), sol) + mul_int(__ldg(t + 7), sol2));
      sol = -ccd_det_int(t, __dmul_rn(__ldg(t + 9), ssi) - __dmul_rn(__ldg(t + 11), si));
      sol2 = ccd_det_int(t, __dmul_rn(__ldg(t + 8), ssi) - __dmul_rn(__ldg(t + 10), si));
      Sl[(int64_t)i * st] = sol;
      SSl[(int64_t)i * st] = sol2;
    }
  }
}

// Few lines: the chain of dependent operations along a line is what takes the
// time (a warp's FP64 instruction takes as long for one line as for 32).  Four
// lanes share a line: each forms one of the four products of a block row and
// the right-hand side of one point of every four, so a point costs the warp
// its chain of 3 + 7 FP64 instructions and 2 for the right-hand side, not 35
// (curvature of 128x256 cells 1.23 ms before, now 0.57).
__global__ void __launch_bounds__(32) k_ccd_lines4(CcdBatch batch) {
  const int pass = blockIdx.y;
  const CcdArgs& c = batch.c[pass];
  const double* __restrict__ table = batch.table[pass];
  const int lines = c.n1 * c.n2;
  const int own = blockIdx.x * 8 + (threadIdx.x >> 2);
  if (blockIdx.x * 8 >= lines) return;  // (whole warps only: lanes exchange values)
  const bool live = own < lines;
  const int r = threadIdx.x & 3;  // the lane's product, and its point of a batch
  const bool odd = r & 1, low = r < 2;
  const int64_t st = c.st;
  const int L = c.L;
  const CcdLine P = ccd_line(batch, c, pass, live ? own : lines - 1);
  const double* __restrict__ fl = P.f;
  double* __restrict__ Sl = P.S;
  double* __restrict__ SSl = P.SS;
  const unsigned all = 0xffffffffu;
  const bool put_s = live && r == 0, put_ss = live && r == 2;
  double s, ss;
  ccd_end(c, fl[0], fl[st], fl[2 * st], fl[3 * st], &s, &ss);
  if (put_s) Sl[0] = s;
  if (put_ss) SSl[0] = ss;
  // f(i-1), f(i), f(i+1) of the lane's point i0 + r, a batch ahead
  double n0, n1, n2;
  const auto load = [&](int i0) {
    const int i = i0 + r < L - 2 ? i0 + r : L - 2;
    n0 = fl[(int64_t)(i - 1) * st];
    n1 = fl[(int64_t)i * st];
    n2 = fl[(int64_t)(i + 1) * st];
  };
  load(1);
  for (int i0 = 1; i0 < L - 1; i0 += 4) {
    const double rs = div_const(c.hd, __dmul_rn(0.9375, n2 - n0));
    const double rss =
        div_const(c.h2d, __fma_rn(-2.0, __dmul_rn(3.0, n1), __dmul_rn(3.0, n0)) + __dmul_rn(3.0, n2));
    load(i0 + 4);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + u;
      if (i >= L - 1) break;
      const double a = __shfl_sync(all, rs, u, 4), b = __shfl_sync(all, rss, u, 4);
      const double m = __dmul_rn(__ldg(table + (size_t)i * kCcdRec + r), odd ? ss : s);
      const double v = (low ? a : b) - (m + __shfl_xor_sync(all, m, 1));
      const double o = __shfl_xor_sync(all, v, 2);
      s = low ? v : o;
      ss = low ? o : v;
      if (put_s) Sl[(int64_t)i * st] = s;
      if (put_ss) SSl[(int64_t)i * st] = ss;
    }
  }
  // back substitution (TWIN_BKS)
  double sol, sol2;
  {
    const int i = L - 1;
    const double* t = table + (size_t)i * kCcdRec;
    double sn, ssn;
    ccd_end(c, fl[(int64_t)i * st], fl[(int64_t)(i - 1) * st], fl[(int64_t)(i - 2) * st],
            fl[(int64_t)(i - 3) * st], &sn, &ssn);
    sn = -sn - (__ldg(t) * s + __ldg(t + 1) * ss);
    ssn = ssn - (__ldg(t + 2) * s + __ldg(t + 3) * ss);
    sol = -ccd_det(t, __ldg(t + 9) * ssn - __ldg(t + 11) * sn);
    sol2 = ccd_det(t, __ldg(t + 8) * ssn - __ldg(t + 10) * sn);
    if (put_s) Sl[(int64_t)i * st] = sol;
    if (put_ss) SSl[(int64_t)i * st] = sol2;
  }
  __syncwarp();  // the lanes read back each other's swept values
  const int k2 = low ? (odd ? 11 : 9) : (odd ? 10 : 8);
  double ns, nss;
  const auto back = [&](int i0) {
    const int i = i0 - r > 0 ? i0 - r : 0;
    ns = Sl[(int64_t)i * st];
    nss = SSl[(int64_t)i * st];
  };
  back(L - 2);
  for (int i0 = L - 2; i0 >= 0; i0 -= 4) {
    const double cs = ns, css = nss;
    back(i0 - 4);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 - u;
      if (i < 0) break;
      const double* t = table + (size_t)i * kCcdRec;
      const double a = __shfl_sync(all, cs, u, 4), b = __shfl_sync(all, css, u, 4);
      double m = __dmul_rn(__ldg(t + 4 + r), odd ? sol2 : sol);
      double v = (low ? a : b) - (m + __shfl_xor_sync(all, m, 1));
      double o = __shfl_xor_sync(all, v, 2);
      // even lanes take ssi = the high pair's value, odd ones si = the low pair's
      m = __dmul_rn(__ldg(t + k2), low == odd ? v : o);
      o = __shfl_xor_sync(all, m, 1);
      v = ccd_det(t, (odd ? o : m) - (odd ? m : o));
      o = __shfl_xor_sync(all, v, 2);
      sol = -(low ? v : o);
      sol2 = low ? o : v;
      if (put_s) Sl[(int64_t)i * st] = sol;
      if (put_ss) SSl[(int64_t)i * st] = sol2;
    }
  }
}

__device__ __forceinline__ int clampi(int x, int n) { return x < 1 ? 1 : (x > n ? n : x); }

// bc: every ghost value is the boundary value of its clamped index (the x,
// y, z passes of copies compose to that).  One warp per padded row; rows
// outside the interior in y or z are done whole, others at their x ghosts.
__global__ void __launch_bounds__(256) k_ccd_bc(NsArgs a, double* f0, double* f1, double* f2,
                                                double* f3) {
  const int g = a.g;
  const bool three = a.nz > 1;
  const int py = a.ny + 2 * g, pz = three ? a.nz + 2 * g : 1;
  const int rows = py * pz;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  double* F[4] = {f0, f1, f2, f3};
  for (int r = warp; r < rows; r += nwarps) {
    const int j = r % py + 1 - g;
    const int k = three ? r / py + 1 - g : 1;
    const bool whole = j < 1 || j > a.ny || (three && (k < 1 || k > a.nz));
    const int cnt = whole ? a.nx + 2 * g : 2 * g;
    const int jc = clampi(j, a.ny), kc = three ? clampi(k, a.nz) : 1;
    for (int t = lane; t < cnt; t += 32) {
      const int i = whole ? t + 1 - g : (t < g ? t + 1 - g : a.nx + 1 + (t - g));
      const int ic = clampi(i, a.nx);
      const int64_t src = (int64_t)(ic - 1) + (int64_t)(jc - 1) * a.sy + (int64_t)(kc - 1) * a.sz;
      const int64_t dst = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if (F[c]) F[c][dst] = F[c][src];
    }
  }
}

// curv on the interior (others_normals.f90 curv): arrays at element (1,1,1)
template <bool kThree>
__global__ void __launch_bounds__(256) k_curvature(NsArgs a, const double* __restrict__ fx_,
                                                   const double* __restrict__ fy_,
                                                   const double* __restrict__ fz_,
                                                   const double* __restrict__ fxx,
                                                   const double* __restrict__ fyy,
                                                   const double* __restrict__ fzz,
                                                   const double* __restrict__ fxy,
                                                   const double* __restrict__ fxz,
                                                   const double* __restrict__ fyz,
                                                   double* __restrict__ curv) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > a.nx || j > a.ny) return;
  const int64_t q = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
  // (products, the root and the quotient on the integer pipes: 14 FP64
  // operations in 3D where the formula takes 33 and a root and a division)
  const double fx = fx_[q], fy = fy_[q];
  const double xx = mul_int(fx, fx), yy = mul_int(fy, fy);
  if (!kThree) {
    const double num = (mul_int(fyy[q], xx) + mul_int(fxx[q], yy)) -
                       mul_int(mul_int(scale2<1>(fxy[q]), fx), fy);
    const double sq = (xx + yy) + 1.0e-12;
    curv[q] = div_int(num, rcp_int(mul_int(sq, sqrt_int(sq))));
  } else {
    const double fz = fz_[q], zz = mul_int(fz, fz);
    const double a2 = fxx[q], b2 = fyy[q], c2 = fzz[q];
    const double num =
        ((mul_int(b2 + c2, xx) + mul_int(a2 + c2, yy)) + mul_int(a2 + b2, zz)) -
        scale2<1>((mul_int(mul_int(fxy[q], fx), fy) + mul_int(mul_int(fxz[q], fx), fz)) +
                  mul_int(mul_int(fyz[q], fy), fz));
    const double sq = ((xx + yy) + zz) + 1.0e-12;
    curv[q] = div_int(num, rcp_int(mul_int(sq, sqrt_int(sq))));
  }
}


// ls_funs at one value (others.f90:1-37): heavy and delta of x = phi/ls_wid
__device__ __forceinline__ void mp_funs(double phi, double ls_wid, double* heavy, double* delta) {
  const double pi = 3.141592653589793;
  const double x = phi / ls_wid;
  double h, hp;
  if (x > 1.0 - 1.0e-12) {
    h = 1.0;
    hp = 0.0;
  } else if (x < -1.0 + 1.0e-12) {
    h = 0.0;
    hp = 0.0;
  } else {
    h = 0.5 * (1.0 + x + sin(pi * x) / pi);
    hp = 0.5 * (1.0 + cos(pi * x)) / ls_wid;
  }
  *heavy = fmax(fmin(h, 1.0), 0.0);
  *delta = hp;
}

// mass_preserving_level_set's sums over the interior (ls_mv's mass and the
// lambda denominator): acc[0] = sum rho H dv, acc[1] = sum delta^2 |grad phi|
// (2 (1 - rho_12) H + rho_12) dv; |grad phi| from the compact gradient.
// Beyond the band (|phi| > out, as bits; ls_outside_bits) H is 0 or 1 and delta
// 0: a cell adds dv or nothing to the first sum and, its gradient being finite,
// nothing to the second.
__device__ __forceinline__ bool mp_outside(long long out, double phi) {
  const long long m = __double_as_longlong(phi) & 0x7fffffffffffffffll;
  return m > out && m <= 0x7ff0000000000000ll;
}

__global__ void __launch_bounds__(kRedThreads) k_mpls_sums(NsArgs a, const double* phi,
                                                           const double* gx, const double* gy,
                                                           const double* gz, double ls_wid,
                                                           long long out, double rho_12,
                                                           double dv, ReduceScratch R) {
  double acc[2] = {0.0, 0.0};
  const int rows = a.ny * a.nz;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const int j = row % a.ny + 1, k = row / a.ny + 1;
    for (int i = threadIdx.x + 1; i <= a.nx; i += blockDim.x) {
      const int64_t q = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
      const double ph = phi[q];
      if (mp_outside(out, ph) &&
          (!gx || max(max(idiv_mag(gx[q]), idiv_mag(gy[q])), gz ? idiv_mag(gz[q]) : 0u) <
                      (1023u + 400u) << 20)) {
        if (__double_as_longlong(ph) >= 0) acc[0] += dv;
        continue;
      }
      double heavy, delta;
      mp_funs(ph, ls_wid, &heavy, &delta);
      const double rho = heavy + rho_12 * (1.0 - heavy);
      acc[0] += rho * heavy * dv;
      if (!gx) continue;  // the mass alone
      const double g2 = gz ? (gx[q] * gx[q] + gy[q] * gy[q]) + gz[q] * gz[q]
                           : gx[q] * gx[q] + gy[q] * gy[q];
      const double grad = sqrt(g2);
      double plam = delta * delta * grad;
      plam = plam * (2.0 * (1.0 - rho_12) * heavy + rho_12) * a.dx * a.dy;
      if (gz) plam = plam * a.dz;
      acc[1] += plam;
    }
  }
  grid_sum_finish<2>(acc, R, kSlotSum);
}

// phi += lam delta |grad phi| on the interior (delta of the phi before)
__global__ void __launch_bounds__(256) k_mpls_update(NsArgs a, double* phi, const double* gx,
                                                     const double* gy, const double* gz,
                                                     double ls_wid, long long out, double lam) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > a.nx || j > a.ny) return;
  const int64_t q = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
  const double ph = phi[q];
  const double x = gx[q], y = gy[q], z = gz ? gz[q] : 0.0;
  if (mp_outside(out, ph) && max(max(idiv_mag(x), idiv_mag(y)), idiv_mag(z)) < (1023u + 400u) << 20)
    return;  // delta = 0
  double heavy, delta;
  mp_funs(ph, ls_wid, &heavy, &delta);
  const double g2 = gz ? (x * x + y * y) + z * z : x * x + y * y;
  phi[q] = ph + lam * delta * sqrt(g2);
}

// vof_wlic_solver's flux along axis ax at faces 0..n of that axis and rows
// 0..n of the others (the reference's is-1..ie ranges): the WLIC blend of the
// THINC flux (beta = 2.3) and the upwind flux by the normal's share, the
// normal being surface_norms2's central difference of phi at the clamped
// upwind cell (zero-gradient ghosts).  Arrays at element (1,1,1).
__global__ void __launch_bounds__(256) k_wlic_flux(NsArgs a, int ax, const double* __restrict__ vof,
                                                   const double* __restrict__ vel,
                                                   const double* __restrict__ phi,
                                                   double* __restrict__ flux) {
  const bool three = a.nz > 1;
  const int i = blockIdx.x * 32 + threadIdx.x;
  const int j = blockIdx.y * 8 + threadIdx.y;
  const int k = three ? (int)blockIdx.z : 1;
  if (i > a.nx || j > a.ny) return;
  const double eps = 1.0e-12, beta = 2.3;
  const double dt = a.dt;
  const double hs[3] = {a.dx, a.dy, a.dz};
  const int n[3] = {a.nx, a.ny, a.nz};
  const int64_t st[3] = {1, a.sy, a.sz};
  const int64_t q = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
  const double u = vel[q];
  int cc[3] = {i, j, k};
  double isgn = 1.0;
  if (!(u > 0.0)) {
    cc[ax] += 1;
    isgn = 0.0;
  }
  const int64_t qi = q + (cc[ax] - (ax == 0 ? i : (ax == 1 ? j : k))) * st[ax];
  const double f = vof[qi];
  double l;
  if (f > 1.0 - eps || f < eps) {
    l = f * u * dt;
  } else {
    const int cb = cc[ax] - 1 < 1 ? 1 : cc[ax] - 1;
    const int64_t qb = qi + (cb - cc[ax]) * st[ax];
    const double alpha = vof[qb] < vof[qi + st[ax]] ? 1.0 : -1.0;
    const double h = hs[ax];
    const double a1 = exp(beta * (2.0 * f - 1.0) / alpha);
    const double a3 = exp(beta);
    const double xc = 0.5 / beta * log((a3 * a3 - a1 * a3) / (a1 * a3 - 1.0));
    const double a4 = cosh(beta * ((isgn - u * dt / h) - xc));
    const double a5 = cosh(beta * (isgn - xc));
    int c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) c[d] = cc[d] < 1 ? 1 : (cc[d] > n[d] ? n[d] : cc[d]);
    if (!three) c[2] = 1;
    const int64_t qc = (int64_t)(c[0] - 1) + (int64_t)(c[1] - 1) * a.sy + (int64_t)(c[2] - 1) * a.sz;
    double nrm[3];
    nrm[0] = 0.5 * (phi[qc + 1] - phi[qc - 1]) / a.dx;
    nrm[1] = 0.5 * (phi[qc + a.sy] - phi[qc - a.sy]) / a.dy;
    nrm[2] = three ? 0.5 * (phi[qc + a.sz] - phi[qc - a.sz]) / a.dz : 0.0;
    double w = three ? (fabs(nrm[0]) + fabs(nrm[1])) + fabs(nrm[2]) : fabs(nrm[0]) + fabs(nrm[1]);
    w = fabs(nrm[ax]) / w;
    l = 0.5 * (u * dt - alpha * h / beta * log(a4 / a5));
    l = l * w + (1.0 - w) * f * u * dt;
  }
  flux[q] = l;
}

// the cell update of one sweep (clipped to [0, 1] after the last sweep)
__global__ void __launch_bounds__(256) k_wlic_update(NsArgs a, int ax, int last, double* vof,
                                                     const double* __restrict__ vof_old,
                                                     const double* __restrict__ vel,
                                                     const double* __restrict__ flux) {
  const int i = blockIdx.x * 32 + threadIdx.x + 1;
  const int j = blockIdx.y * 8 + threadIdx.y + 1;
  const int k = blockIdx.z + 1;
  if (i > a.nx || j > a.ny) return;
  const double eps = 1.0e-12;
  const int64_t st = ax == 0 ? 1 : (ax == 1 ? a.sy : a.sz);
  const double h = ax == 0 ? a.dx : (ax == 1 ? a.dy : a.dz);
  const int64_t q = (int64_t)(i - 1) + (int64_t)(j - 1) * a.sy + (int64_t)(k - 1) * a.sz;
  double f = vof[q] - (flux[q] - flux[q - st]) / h + vof_old[q] * a.dt * (vel[q] - vel[q - st]) / h;
  if (last) {
    if (f < eps) f = 0.0;
    if (f > 1.0 - eps) f = 1.0;
  }
  vof[q] = f;
}
}  // namespace

void launch_ccd_lines(cudaStream_t s, const CcdBatch& b) {
  int lines = 0, all = 0;
  for (int i = 0; i < b.n; ++i) {
    lines = std::max(lines, b.c[i].n1 * b.c[i].n2);
    all += b.c[i].n1 * b.c[i].n2;
  }
  if (all >= kCcdManyLines)
    k_ccd_lines<<<dim3((unsigned)((lines + kCcdThreads - 1) / kCcdThreads), (unsigned)b.n),
                  kCcdThreads, 0, s>>>(b);
  else  // one warp per block: the few warps spread over the SMs
    k_ccd_lines4<<<dim3((unsigned)((lines + 7) / 8), (unsigned)b.n), 32, 0, s>>>(b);
}

void launch_ccd_bc(cudaStream_t s, const NsArgs& a, double* const f[4]) {
  const int pz = a.nz > 1 ? a.nz + 2 * a.g : 1;
  const long rows = (long)(a.ny + 2 * a.g) * pz;
  const unsigned blocks = (unsigned)std::min<long>((rows + 7) / 8, 152L * 16);
  k_ccd_bc<<<blocks, 256, 0, s>>>(a, f[0], f[1], f[2], f[3]);
}

void launch_curvature(cudaStream_t s, const NsArgs& a, const double* const d1[3],
                      const double* const d2[6], double* curv) {
  const dim3 block(32, 8);
  const dim3 grid((unsigned)((a.nx + 31) / 32), (unsigned)((a.ny + 7) / 8), (unsigned)a.nz);
  if (a.nz > 1)
    k_curvature<true><<<grid, block, 0, s>>>(a, d1[0], d1[1], d1[2], d2[0], d2[1], d2[2], d2[3],
                                             d2[4], d2[5], curv);
  else
    k_curvature<false><<<grid, block, 0, s>>>(a, d1[0], d1[1], nullptr, d2[0], d2[1], nullptr,
                                              d2[3], nullptr, nullptr, curv);
}

void launch_mpls_sums(cudaStream_t s, const NsArgs& a, const double* phi, const double* const g[3],
                      double ls_wid, double rho_12, double dv, const ReduceScratch& R) {
  const int blocks = std::min(reduce_blocks_for((size_t)a.ny * a.nz), R.max_blocks);
  const long long out = std::isfinite(rho_12) ? ls_outside_bits(ls_wid) : 0x7fffffffffffffffll;
  k_mpls_sums<<<blocks, kRedThreads, 0, s>>>(a, phi, g[0], g[1], g[2], ls_wid, out, rho_12, dv, R);
}

void launch_mpls_update(cudaStream_t s, const NsArgs& a, double* phi, const double* const g[3],
                        double ls_wid, double lam) {
  const dim3 block(32, 8);
  const dim3 grid((unsigned)((a.nx + 31) / 32), (unsigned)((a.ny + 7) / 8), (unsigned)a.nz);
  const long long out = std::isfinite(lam) ? ls_outside_bits(ls_wid) : 0x7fffffffffffffffll;
  k_mpls_update<<<grid, block, 0, s>>>(a, phi, g[0], g[1], g[2], ls_wid, out, lam);
}

void launch_wlic(cudaStream_t s, const NsArgs& a, int ax, double* vof, const double* vof_old,
                 const double* vel, const double* phi, double* flux) {
  const dim3 block(32, 8);
  const bool three = a.nz > 1;
  const dim3 gf((unsigned)((a.nx + 1 + 31) / 32), (unsigned)((a.ny + 1 + 7) / 8),
                (unsigned)(three ? a.nz + 1 : 1));
  k_wlic_flux<<<gf, block, 0, s>>>(a, ax, vof, vel, phi, flux);
  const dim3 gu((unsigned)((a.nx + 31) / 32), (unsigned)((a.ny + 7) / 8), (unsigned)a.nz);
  k_wlic_update<<<gu, block, 0, s>>>(a, ax, ax == (three ? 2 : 1), vof, vof_old, vel, flux);
}

}  // namespace gbmg
