// The bottom of the V-cycle in one thread block (sm_103a).
//
// Levels with at most kSubMaxCells cells are launch-latency bound: a sweep of
// 16^3 cells is a few microseconds of launch and drain for nanoseconds of
// work.  This kernel runs everything from level lc down and back up --
// sweeps, residual + restriction, the dense coarsest solve, prolongation --
// in one block, with every level's unknown, right-hand side and face
// coefficients and the coarsest matrices in shared memory.  Phases are
// separated by __syncthreads().  Each step does the arithmetic of the
// corresponding separate kernel in the same order (red-black update, children
// summed in z, y, x order, slopes added x, y, z), so the cycle is the same cycle.
//
// One block is bound by the instructions and the latency of its phases (from
// 16^3 down it had been 68,000 cycles, 35 us), so:
//   - the coefficients and matrices, which no kernel of the cycle writes, are
//     staged before the wait for the preceding kernel;
//   - arrays are padded with zeros by a plane (2D: a row) and a wall's
//     coefficient is a stored zero, so a stencil has no bounds tests: a term
//     that the separate kernels leave out adds an exact zero here;
//   - a thread's cells of a level are worked out once for all sweeps, by
//     products with reciprocals; it relaxes two cells at once and in FP32
//     keeps their coefficients in registers, loaded for both cells of an x pair
//     together (a colour's cells alone are two apart: two passes per read);
//   - warps without cells of a level neither load nor relax (on 8^3 their idle
//     loads took 1,500 of a sweep's 4,200 cycles);
//   - the residuals of all fine cells are formed in parallel, then summed per
//     coarse cell in order, and the slopes of the prolongation once per coarse
//     cell and applied per x pair;
//   - a row of the coarsest products is read down its column, conflict-free
//     (both matrices are symmetric bit for bit); in FP64 eight threads share a
//     row and the residual takes the operator's seven values for the dense row.
// Cycles after the wait, before the last three -> now: FP32 from 16^3 down
// 39,900 -> 30,700 (sweeps of 16^3 7,700 -> 6,000 each way, of 8^3 4,200 ->
// 2,500, restriction 4,100 -> 2,900), FP32 from 32^2 down 26,000 -> 18,700,
// FP64 from 16^2 down 30,400 -> 20,100 (the coarsest solve 14,300 -> 6,300).
// Levels kept colour-split relax 16^3 faster, but lose that again in the
// restriction, the prolongation and the stores out.
#include "gbmg_internal.h"
#include "mg_cells.cuh"
#include "pdl.cuh"

namespace gbmg {

namespace {

constexpr int kSubThreads = 1024;
// the FP64 levels carry 1/diagonal, the FP32 levels divide
template <typename T>
constexpr bool kSubIdiag = sizeof(T) == 8;

// Neighbour sum and diagonal of cell q (x-, x+, y-, y+, z-, z+)
template <typename T>
__device__ __forceinline__ void sub_stencil(const SubLevel<T>& L, const T* __restrict__ p, int q,
                                            T& s, T& d) {
  const int sy = L.nx, sz = L.nx * L.ny;
  T c;
  s = T(0);
  c = L.cx[q]; s += c * p[q - 1]; d = c;
  c = L.cx[q + 1]; s += c * p[q + 1]; d += c;
  c = L.cy[q]; s += c * p[q - sy]; d += c;
  c = L.cy[q + sy]; s += c * p[q + sy]; d += c;
  if (L.nz > 1) {
    c = L.cz[q]; s += c * p[q - sz]; d += c;
    c = L.cz[q + sz]; s += c * p[q + sz]; d += c;
  }
}

// t / d for t * d < 2^32 (r = ceil(2^32 / d), 0 for d = 1)
__device__ __forceinline__ int sub_div(int t, unsigned r) {
  return r ? (int)__umulhi((unsigned)t, r) : t;
}

// (i, j, k) of cell q
template <typename T>
__device__ __forceinline__ void sub_ijk(const SubLevel<T>& L, int q, int& i, int& j, int& k) {
  const int row = sub_div(q, L.rx);
  i = q - row * L.nx;
  k = sub_div(row, L.ry);
  j = row - k * L.ny;
}

// x pair t of a level: its first cell, the colour of that cell, and whether the
// pair has a second one; first = -1 beyond the last pair
struct SubPair {
  int first, colour;
  bool two;
  // the pair's cell of a colour, or -1
  __device__ __forceinline__ int cell(int c) const {
    return first < 0 || (colour != c && !two) ? -1 : first + (colour ^ c);
  }
};

template <typename T>
__device__ __forceinline__ SubPair sub_pair(const SubLevel<T>& L, int t) {
  const int hx = (L.nx + 1) >> 1;
  if (t >= hx * L.ny * L.nz) return SubPair{-1, 0, false};
  const int row = sub_div(t, L.rh), m = t - row * hx;
  const int k = sub_div(row, L.ry), j = row - k * L.ny;
  return SubPair{row * L.nx + 2 * m, (j + k) & 1, 2 * m + 1 < L.nx};
}

// the relaxed value of one cell
template <typename T>
__device__ __forceinline__ T sub_relax(const SubLevel<T>& L, const T* sol, const T* src, int q,
                                       bool zero) {
  T s, d;
  if constexpr (kSubIdiag<T>) {
    s = T(0);
    if (!zero) sub_stencil(L, sol, q, s, d);
    return (s - src[q]) * L.id[q];
  } else {
    sub_stencil(L, sol, q, s, d);
    if (zero) s = T(0);  // (the level's values are taken as zero)
    return (s - src[q]) / d;
  }
}

// A cell's constants of a sweep in registers (FP32): a colour's cells are two
// apart, so every shared-memory read of a colour launch takes two passes, and
// the six coefficients and b are most of the thirteen a cell would read
template <typename T>
struct SubCell {
  T c[6], b;
};

// the two cells of a pair (nx even), the one of colour `first` in u[0]; two at a
// time from shared memory
template <typename T>
__device__ __forceinline__ void sub_load(const SubLevel<T>& L, const T* src, const SubPair& p,
                                         int first, SubCell<T> (&u)[2]) {
  using V2 = typename cells::Vec2<T>::type;
  const auto two = [](const T* a) { return *reinterpret_cast<const V2*>(a); };
  const int q = p.first, sy = L.nx, sz = L.nx * L.ny;
  const V2 x = two(L.cx + q), ym = two(L.cy + q), yp = two(L.cy + q + sy), b = two(src + q);
  const T xr = L.cx[q + 2];
  V2 zm{T(0), T(0)}, zp{T(0), T(0)};
  if (L.nz > 1) {
    zm = two(L.cz + q);
    zp = two(L.cz + q + sz);
  }
  const bool swap = p.colour != first;
  const auto put = [&](SubCell<T>& v, bool second) {
    v.c[0] = second ? x.y : x.x;
    v.c[1] = second ? xr : x.y;
    v.c[2] = second ? ym.y : ym.x;
    v.c[3] = second ? yp.y : yp.x;
    v.c[4] = second ? zm.y : zm.x;
    v.c[5] = second ? zp.y : zp.x;
    v.b = second ? b.y : b.x;
  };
  put(u[0], swap);
  put(u[1], !swap);
}

// sub_relax from the registers
template <typename T>
__device__ __forceinline__ T sub_relax(const SubLevel<T>& L, const T* p, const SubCell<T>& u,
                                       bool zero) {
  const int sy = L.nx, sz = L.nx * L.ny;
  T s = T(0), d = u.c[0];
  s += u.c[0] * p[-1];
  s += u.c[1] * p[1]; d += u.c[1];
  s += u.c[2] * p[-sy]; d += u.c[2];
  s += u.c[3] * p[sy]; d += u.c[3];
  if (L.nz > 1) {
    s += u.c[4] * p[-sz]; d += u.c[4];
    s += u.c[5] * p[sz]; d += u.c[5];
  }
  if (zero) s = T(0);  // (the level's values are taken as zero)
  return (s - u.b) / d;
}

// n red-black sweeps on a shared-memory level; zero: from a zero guess.  Only
// warps with cells of a level load and relax: on the small levels the others'
// idle loads took longer than the sweeps.
template <typename T>
__device__ void sub_sweeps(const SubLevel<T>& L, T* sol, const T* src, int n, int first, bool zero) {
  const int npair = ((L.nx + 1) >> 1) * L.ny * L.nz;
  if (kSubIdiag<T> || (L.nx & 1) || npair > 2 * kSubThreads) {
    const SubPair a = sub_pair(L, (int)threadIdx.x);
    for (int it = 0; it < 2 * n; ++it) {
      const int color = first ^ (it & 1);
      const bool z = zero && it == 0;
      const int q = a.cell(color);
      if (q >= 0) sol[q] = sub_relax(L, sol, src, q, z);
      for (int t = threadIdx.x + kSubThreads; t < npair; t += kSubThreads) {
        const int r = sub_pair(L, t).cell(color);
        if (r >= 0) sol[r] = sub_relax(L, sol, src, r, z);
      }
      __syncthreads();
    }
    return;
  }
  const int ta = (int)threadIdx.x, tb = ta + kSubThreads;
  const bool has_a = ta < npair, has_b = tb < npair;
  SubCell<T> ua[2], ub[2];  // [colour of the sweep]
  SubPair a{0, 0, true}, b{0, 0, true};
  if (has_a && n > 0) {
    a = sub_pair(L, ta);
    sub_load(L, src, a, first, ua);
  }
  if (has_b && n > 0) {
    b = sub_pair(L, tb);
    sub_load(L, src, b, first, ub);
  }
  for (int it = 0; it < n; ++it)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const bool z = zero && it == 0 && c == 0;
      T* pa = sol + a.first + (a.colour ^ first ^ c);
      T* pb = sol + b.first + (b.colour ^ first ^ c);
      if (has_b) {
        const T va = sub_relax(L, pa, ua[c], z), vb = sub_relax(L, pb, ub[c], z);
        *pa = va;
        *pb = vb;
      } else if (has_a) {
        *pa = sub_relax(L, pa, ua[c], z);
      }
      __syncthreads();
    }
}

// coarse src = mean of the children's residuals (fine -> coarse, shared
// memory); half (FP64, as restrict_cell): the children of colour 1, relaxed
// last, have none.  res: one value per fine cell.
template <typename T>
__device__ void sub_restrict(const SubLevel<T>& F, const T* fsol, const T* fsrc,
                             const SubLevel<T>& C, T* csrc, T* res, bool half) {
  const bool skip = sizeof(T) == 8 && half;
  // (a thread per pair where only one of its cells counts)
  const int nf = skip ? ((F.nx + 1) >> 1) * F.ny * F.nz : F.nx * F.ny * F.nz;
  for (int t = threadIdx.x; t < nf; t += kSubThreads) {
    const int q = skip ? sub_pair(F, t).cell(0) : t;
    if (q < 0) continue;
    T s, d;
    sub_stencil(F, fsol, q, s, d);
    res[q] = fsrc[q] - (s - d * fsol[q]);
  }
  __syncthreads();
  const int n = C.nx * C.ny * C.nz;
  for (int cq = threadIdx.x; cq < n; cq += kSubThreads) {
    int I, J, K;
    sub_ijk(C, cq, I, J, K);
    T acc = T(0);
    if (sizeof(T) == 4 && F.fx == 2) {
      using V2 = typename cells::Vec2<T>::type;
      const T* r = res + (F.fz * K * F.ny + F.fy * J) * F.nx + 2 * I;
      const int sy = F.fy == 2 ? F.nx : 0, sz = F.fz == 2 ? F.nx * F.ny : 0;
      V2 v[4];
      v[0] = *reinterpret_cast<const V2*>(r);
      v[1] = *reinterpret_cast<const V2*>(r + sy);
      v[2] = *reinterpret_cast<const V2*>(r + sz);
      v[3] = *reinterpret_cast<const V2*>(r + sz + sy);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (((c & 1) && F.fy == 1) || ((c & 2) && F.fz == 1)) continue;
        acc += v[c].x;
        acc += v[c].y;
      }
      csrc[cq] = acc * F.mean;
      continue;
    }
    for (int dz = 0; dz < F.fz; ++dz)
      for (int dy = 0; dy < F.fy; ++dy)
        for (int dx = 0; dx < F.fx; ++dx) {
          const int i = F.fx * I + dx, j = F.fy * J + dy, k = F.fz * K + dz;
          if (skip && ((i + j + k) & 1)) continue;
          acc += res[(k * F.ny + j) * F.nx + i];
        }
    csrc[cq] = acc * F.mean;
  }
  __syncthreads();
}

// fine sol += central-slope interpolation of the coarse sol; m: a value
// per coarse cell and axis (FP64: live >= 0, the cells of that colour only)
template <typename T>
__device__ void sub_prolong(const SubLevel<T>& F, T* fsol, const SubLevel<T>& C, const T* e, T* m,
                            int live) {
  const int nc = C.nx * C.ny * C.nz;
  const int csy = C.nx, csz = C.nx * C.ny;
  // a quarter of the slope along each coarsened axis, axis after axis
  T* my = m + (F.fx == 2 ? nc : 0);
  T* mz = my + (F.fy == 2 ? nc : 0);
  for (int cq = threadIdx.x; cq < nc; cq += kSubThreads) {
    int I, J, K;
    sub_ijk(C, cq, I, J, K);
    const T ec = e[cq];
    if (F.fx == 2)
      m[cq] = T(0.25) * (T(0.5) * ((I < C.nx - 1 ? e[cq + 1] : ec) - (I > 0 ? e[cq - 1] : ec)));
    if (F.fy == 2)
      my[cq] = T(0.25) * (T(0.5) * ((J < C.ny - 1 ? e[cq + csy] : ec) - (J > 0 ? e[cq - csy] : ec)));
    if (F.fz == 2)
      mz[cq] =
          T(0.25) * (T(0.5) * ((K < C.nz - 1 ? e[cq + csz] : ec) - (K > 0 ? e[cq - csz] : ec)));
  }
  __syncthreads();
  const int n = F.nx * F.ny * F.nz;
  if (sizeof(T) == 4 && F.fx == 2) {
    // the two cells of a pair share their coarse cell
    using V2 = typename cells::Vec2<T>::type;
#pragma unroll 2
    for (int t = threadIdx.x; t < n / 2; t += kSubThreads) {
      const int row = sub_div(t, F.rh), I = t - row * C.nx;
      const int k = sub_div(row, F.ry), j = row - k * F.ny;
      const int cq = ((k >> (F.fz - 1)) * C.ny + (j >> (F.fy - 1))) * C.nx + I;
      V2* o = reinterpret_cast<V2*>(fsol) + t;
      const T ec = e[cq], mx = m[cq];
      V2 v = *o;
      T v0 = ec + -mx, v1 = ec + mx;
      if (F.fy == 2) {
        const T y = (j & 1) ? my[cq] : -my[cq];
        v0 += y;
        v1 += y;
      }
      if (F.fz == 2) {
        const T z = (k & 1) ? mz[cq] : -mz[cq];
        v0 += z;
        v1 += z;
      }
      v.x += v0;
      v.y += v1;
      *o = v;
    }
    __syncthreads();
    return;
  }
  const bool one = sizeof(T) == 8 && live >= 0;
  const int nt = one ? ((F.nx + 1) >> 1) * F.ny * F.nz : n;
#pragma unroll 2
  for (int t = threadIdx.x; t < nt; t += kSubThreads) {
    const int q = one ? sub_pair(F, t).cell(live) : t;
    if (q < 0) continue;
    int i, j, k;
    sub_ijk(F, q, i, j, k);
    const int cq = ((k >> (F.fz - 1)) * C.ny + (j >> (F.fy - 1))) * C.nx + (i >> (F.fx - 1));
    T val = e[cq];
    if (F.fx == 2) val += (i & 1) ? m[cq] : -m[cq];
    if (F.fy == 2) val += (j & 1) ? my[cq] : -my[cq];
    if (F.fz == 2) val += (k & 1) ? mz[cq] : -mz[cq];
    fsol[q] += val;
  }
  __syncthreads();
}

// sum_q a[q n + t] x[q], added to (sign 1) or taken from (sign -1) acc, in order,
// as k_coarse_solve
template <typename T, int kSign>
__device__ __forceinline__ T sub_row(int n, const T* a, const T* x, int t, T acc) {
#pragma unroll 16
  for (int q = 0; q < n; ++q) {
    if (kSign > 0) acc += a[q * n + t] * x[q];
    else acc -= a[q * n + t] * x[q];
  }
  return acc;
}

// sum_q a[q n + t] x[q] for every row t (FP64), the result with the first n
// threads.  One thread per row waits out the latency of each addition; here row
// t & 63 is shared by kSubParts threads with two partial sums each, and the parts
// meet in shared memory.
constexpr int kSubParts = 8;
__device__ __forceinline__ double sub_rows(int n, const double* a, const double* x, double* part) {
  const int t = threadIdx.x & (kMaxCoarse - 1), g = threadIdx.x / kMaxCoarse;
  if (g < kSubParts && t < n) {
    double p0 = 0.0, p1 = 0.0;
    int q = g;
#pragma unroll 4
    for (; q + kSubParts < n; q += 2 * kSubParts) {
      p0 += a[q * n + t] * x[q];
      p1 += a[(q + kSubParts) * n + t] * x[q + kSubParts];
    }
    if (q < n) p0 += a[q * n + t] * x[q];
    part[g * kMaxCoarse + t] = p0 + p1;
  }
  __syncthreads();
  double v = 0.0;
  if (threadIdx.x < n) {
    double u[kSubParts];
#pragma unroll
    for (int i = 0; i < kSubParts; ++i) u[i] = part[i * kMaxCoarse + t];
#pragma unroll
    for (int w = kSubParts / 2; w > 0; w >>= 1)
#pragma unroll
      for (int i = 0; i < w; ++i) u[i] += u[i + w];
    v = u[0];
  }
  return v;
}

// x = Minv b, one refinement step when max|b - A x| > 1e-10, mean projection
// (as k_coarse_solve); minv and a in shared memory, both symmetric
template <typename T>
__device__ void sub_coarse(const SubLevel<T>& C, int n, const T* minv, const T* a, const T* b, T* x,
                           T* se) {
  const int t = threadIdx.x;
  if constexpr (sizeof(T) == 8) {
    double* part = se + kMaxCoarse;
    const double x0 = sub_rows(n, minv, b, part);
    if (t < n) x[t] = x0;
    __syncthreads();
    int bad = 0;
    if (t < n) {
      // (the rows of A hold at most seven values)
      double s, d;
      sub_stencil(C, x, t, s, d);
      const double e = b[t] - (s - d * x0);
      se[t] = e;
      bad = fabs(e) > 1e-10;
    }
    if (__syncthreads_or(bad)) {
      const double dx = sub_rows(n, minv, se, part);
      if (t < n) x[t] = x0 + dx;
      __syncthreads();
    }
  } else {
    if (t < n) x[t] = sub_row<T, 1>(n, minv, b, t, T(0));
    __syncthreads();
    int bad = 0;
    if (t < n) {
      const T e = sub_row<T, -1>(n, a, x, t, b[t]);
      se[t] = e;
      bad = fabs((double)e) > 1e-10;
    }
    if (__syncthreads_or(bad)) {
      if (t < n) x[t] += sub_row<T, 1>(n, minv, se, t, T(0));
      __syncthreads();
    }
  }
  // the mean: FP32 summed in index order by every thread that needs it, FP64
  // by a tree in each of their warps
  T xv = T(0);
  if (t < kMaxCoarse) {
    T s = T(0);
    if constexpr (sizeof(T) == 8) {
      const int lane = t & 31;
      s = (lane < n ? x[lane] : T(0)) + (lane + 32 < n ? x[lane + 32] : T(0));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    } else if (t < n) {
#pragma unroll 16
      for (int q = 0; q < n; ++q) s += x[q];
    }
    if (t < n) xv = x[t] - s / T(n);
  }
  __syncthreads();
  if (t < n) x[t] = xv;
  __syncthreads();
}

// Shared memory per level (pad = SubLevel::pad zeros): pad, sol, pad, src, then
// each face-coefficient array followed by pad, and 1/diagonal where there is
// one; after the levels one value per cell of the finest one (residuals,
// slopes), the coarsest level's two matrices and its scratch.
template <typename T>
__device__ void subcycle_body(const SubCycle<T>& S, T* base) {
  const int nl = S.nlev;
  const auto cells = [&](int l) { return S.lv[l].nx * S.lv[l].ny * S.lv[l].nz; };
  T* res = base + S.off[nl];
  T* minv = res + cells(0);
  T* adense = minv + S.n_coarse * S.n_coarse;
  T* scratch = adense + S.n_coarse * S.n_coarse;
  const int tid = threadIdx.x;
  for (int l = 0; l < nl; ++l) {
    const int n = cells(l), pad = S.lv[l].pad, na = n + pad;
    T* c = base + S.lv[l].at_c;
#pragma unroll 4
    for (int q = tid; q < n; q += kSubThreads) {
      c[q] = S.lv[l].cx[q];
      c[na + q] = S.lv[l].cy[q];
      c[2 * na + q] = S.lv[l].cz[q];
      if (kSubIdiag<T>) c[3 * na + q] = S.lv[l].id[q];
    }
    for (int q = tid; q < pad; q += kSubThreads)
      c[n + q] = c[na + n + q] = c[2 * na + n + q] = T(0);
    for (int q = tid; q < n + 2 * pad; q += kSubThreads) base[S.off[l] + q] = T(0);
  }
  for (int q = tid; q < S.n_coarse * S.n_coarse; q += kSubThreads) {
    minv[q] = S.minv[q];
    adense[q] = S.adense[q];
  }
  const auto sol = [&](int l) { return base + S.lv[l].at_sol; };
  const auto src = [&](int l) { return base + S.lv[l].at_src; };
  // level l with its coefficients in shared memory
  const auto lv = [&](int l) {
    SubLevel<T> L = S.lv[l];
    const int na = L.at_na;
    const T* c = base + L.at_c;
    L.cx = c;
    L.cy = c + na;
    L.cz = c + 2 * na;
    if (kSubIdiag<T>) L.id = c + 3 * na;
    return L;
  };
  // The set-up kernels that wrote the above are ordinary launches, complete
  // before any kernel of the cycle starts; what follows is the cycle's.
  pdl_wait();
  {
    T* b = src(0);
#pragma unroll 4
    for (int q = tid; q < cells(0); q += kSubThreads) b[q] = __ldcg(S.src_in + q);
  }
  __syncthreads();
  for (int l = 0; l < nl - 1; ++l) {
    const SubLevel<T> L = lv(l);
    sub_sweeps(L, sol(l), src(l), S.nu1, 0, true);
    sub_restrict(L, sol(l), src(l), lv(l + 1), src(l + 1), res, S.nu1 > 0);
  }
  sub_coarse(lv(nl - 1), S.n_coarse, minv, adense, src(nl - 1), sol(nl - 1), scratch);
  for (int l = nl - 2; l >= 0; --l) {
    const SubLevel<T> L = lv(l);
    sub_prolong(L, sol(l), lv(l + 1), sol(l + 1), res, S.nu2 > 0 ? (S.reverse ? 0 : 1) : -1);
    sub_sweeps(L, sol(l), src(l), S.nu2, S.reverse ? 1 : 0, false);
  }
  for (int q = tid; q < cells(0); q += kSubThreads) S.sol_out[q] = sol(0)[q];
}

template <typename T>
__global__ void __launch_bounds__(kSubThreads, 1) k_subcycle(SubCycle<T> S) {
  pdl_launch();
  extern __shared__ __align__(16) unsigned char sub_raw[];
  subcycle_body(S, reinterpret_cast<T*>(sub_raw));
}

}  // namespace

template <typename T>
size_t subcycle_smem(const SubCycle<T>& S) {
  const int n0 = S.lv[0].nx * S.lv[0].ny * S.lv[0].nz;
  return (size_t)(S.off[S.nlev] + n0 + 2 * S.n_coarse * S.n_coarse +
                  (kSubIdiag<T> ? 1 + kSubParts : 1) * kMaxCoarse) * sizeof(T);
}

// The attribute belongs to the kernel, not to a handle: every handle sets the same
// limit (with its own need, a later and smaller handle took the launch from an
// earlier one: invalid argument).
template <typename T>
int subcycle_init(size_t smem) {
  return smem <= kSubMaxSmem &&
                 cudaFuncSetAttribute(k_subcycle<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSubMaxSmem) == cudaSuccess
             ? 0
             : -1;
}

template <typename T>
void launch_subcycle(cudaStream_t s, const SubCycle<T>& S) {
  launch_pdl(k_subcycle<T>, dim3(1), dim3(kSubThreads), subcycle_smem(S), s, S);
}

template size_t subcycle_smem<float>(const SubCycle<float>&);
template size_t subcycle_smem<double>(const SubCycle<double>&);
template int subcycle_init<float>(size_t);
template int subcycle_init<double>(size_t);
template void launch_subcycle<float>(cudaStream_t, const SubCycle<float>&);
template void launch_subcycle<double>(cudaStream_t, const SubCycle<double>&);

}  // namespace gbmg
