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
// 16^3 down 68,000 cycles before, 35 us), so:
//   - the coefficients and matrices, which no kernel of the cycle writes, are
//     staged before the wait for the preceding kernel;
//   - arrays are padded with zeros by a plane (2D: a row) and a wall's
//     coefficient is a stored zero, so a stencil has no bounds tests: a term
//     that the separate kernels leave out adds an exact zero here;
//   - a thread's cells of a level are worked out once for all sweeps, by
//     products with reciprocals; it relaxes two cells at once and in FP32
//     keeps their coefficients in registers;
//   - the residuals of all fine cells are formed in parallel, then summed per
//     coarse cell in order, and the slopes of the prolongation once per coarse
//     cell;
//   - a row of the coarsest products is read down its column, conflict-free
//     (both matrices are symmetric bit for bit).
// With these the block from 16^3 down takes 39,000 cycles after the wait:
// sweeps of 16^3 7,700 of them down and up, the restriction 3,600 (7,500
// before), the coarsest solve 3,800 (21,900), the prolongation 2,900.  Levels
// kept colour-split relax 16^3 in 5,700, but lose that again in the restriction,
// the prolongation and the stores out.
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
  int q;  // -1: no such cell
};

template <typename T>
__device__ __forceinline__ SubCell<T> sub_load(const SubLevel<T>& L, const T* src, int q) {
  SubCell<T> u;
  u.q = q;
  const int r = q < 0 ? 0 : q;
  const int sy = L.nx, sz = L.nx * L.ny;
  u.c[0] = L.cx[r];
  u.c[1] = L.cx[r + 1];
  u.c[2] = L.cy[r];
  u.c[3] = L.cy[r + sy];
  u.c[4] = L.nz > 1 ? L.cz[r] : T(0);
  u.c[5] = L.nz > 1 ? L.cz[r + sz] : T(0);
  u.b = src[r];
  return u;
}

// sub_relax from the registers
template <typename T>
__device__ __forceinline__ T sub_relax(const SubLevel<T>& L, const T* sol, const SubCell<T>& u,
                                       bool zero) {
  const int sy = L.nx, sz = L.nx * L.ny;
  const T* p = sol + u.q;
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

// n red-black sweeps on a shared-memory level; zero: from a zero guess
template <typename T>
__device__ void sub_sweeps(const SubLevel<T>& L, T* sol, const T* src, int n, int first, bool zero) {
  const int npair = ((L.nx + 1) >> 1) * L.ny * L.nz;
  const SubPair a = sub_pair(L, (int)threadIdx.x), b = sub_pair(L, (int)threadIdx.x + kSubThreads);
  const auto rest = [&](int color, bool z) {
    for (int t = threadIdx.x + 2 * kSubThreads; t < npair; t += kSubThreads) {
      const int q = sub_pair(L, t).cell(color);
      if (q >= 0) sol[q] = sub_relax(L, sol, src, q, z);
    }
    __syncthreads();
  };
  if constexpr (kSubIdiag<T>) {
    for (int it = 0; it < 2 * n; ++it) {
      const int color = first ^ (it & 1);
      const bool z = zero && it == 0;
      const int qa = a.cell(color), qb = b.cell(color);
      T va = T(0), vb = T(0);
      if (qa >= 0) va = sub_relax(L, sol, src, qa, z);
      if (qb >= 0) vb = sub_relax(L, sol, src, qb, z);
      if (qa >= 0) sol[qa] = va;
      if (qb >= 0) sol[qb] = vb;
      rest(color, z);
    }
  } else if (n > 0) {
    SubCell<T> u[2][2];  // [colour of the sweep][pair]
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      u[c][0] = sub_load(L, src, a.cell(first ^ c));
      u[c][1] = sub_load(L, src, b.cell(first ^ c));
    }
    for (int it = 0; it < n; ++it)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const bool z = zero && it == 0 && c == 0;
        T va = T(0), vb = T(0);
        if (u[c][0].q >= 0) va = sub_relax(L, sol, u[c][0], z);
        if (u[c][1].q >= 0) vb = sub_relax(L, sol, u[c][1], z);
        if (u[c][0].q >= 0) sol[u[c][0].q] = va;
        if (u[c][1].q >= 0) sol[u[c][1].q] = vb;
        rest(first ^ c, z);
      }
  }
}

// coarse src = mean of the children's residuals (fine -> coarse, shared
// memory); half (FP64, as restrict_cell): the children of colour 1, relaxed
// last, have none.  res: one value per fine cell.
template <typename T>
__device__ void sub_restrict(const SubLevel<T>& F, const T* fsol, const T* fsrc,
                             const SubLevel<T>& C, T* csrc, T* res, bool half) {
  const bool skip = sizeof(T) == 8 && half;
  const int nf = F.nx * F.ny * F.nz;
  for (int q = threadIdx.x; q < nf; q += kSubThreads) {
    if (skip) {
      int i, j, k;
      sub_ijk(F, q, i, j, k);
      if ((i + j + k) & 1) continue;
    }
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
#pragma unroll 2
  for (int q = threadIdx.x; q < n; q += kSubThreads) {
    int i, j, k;
    sub_ijk(F, q, i, j, k);
    if (sizeof(T) == 8 && live >= 0 && ((i + j + k) & 1) != live) continue;
    const int cq = ((k >> (F.fz - 1)) * C.ny + (j >> (F.fy - 1))) * C.nx + (i >> (F.fx - 1));
    T val = e[cq];
    if (F.fx == 2) val += (i & 1) ? m[cq] : -m[cq];
    if (F.fy == 2) val += (j & 1) ? my[cq] : -my[cq];
    if (F.fz == 2) val += (k & 1) ? mz[cq] : -mz[cq];
    fsol[q] += val;
  }
  __syncthreads();
}

// sum_q a[q n + t] x[q], added to (sign 1) or taken from (sign -1) acc.  FP32:
// in order, as k_coarse_solve.  FP64: four partial sums (a chain of dependent
// FP64 operations waits longer than the pipe needs for four).
template <typename T, int kSign>
__device__ __forceinline__ T sub_row(int n, const T* a, const T* x, int t, T acc) {
  if constexpr (sizeof(T) == 8) {
    T p[4] = {acc, T(0), T(0), T(0)};
    int q = 0;
    for (; q + 4 <= n; q += 4)
#pragma unroll
      for (int u = 0; u < 4; ++u) p[u] += (kSign > 0 ? a[(q + u) * n + t] : -a[(q + u) * n + t]) * x[q + u];
    for (; q < n; ++q) p[0] += (kSign > 0 ? a[q * n + t] : -a[q * n + t]) * x[q];
    return (p[0] + p[1]) + (p[2] + p[3]);
  } else {
#pragma unroll 16
    for (int q = 0; q < n; ++q) {
      if (kSign > 0) acc += a[q * n + t] * x[q];
      else acc -= a[q * n + t] * x[q];
    }
    return acc;
  }
}

// x = Minv b, one refinement step when max|b - A x| > 1e-10, mean projection
// (as k_coarse_solve); minv and a in shared memory, both symmetric
template <typename T>
__device__ void sub_coarse(int n, const T* minv, const T* a, const T* b, T* x, T* se) {
  const int t = threadIdx.x;
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
  const auto sol = [&](int l) { return base + S.off[l] + S.lv[l].pad; };
  const auto src = [&](int l) { return base + S.off[l] + cells(l) + 2 * S.lv[l].pad; };
  T* res = base + S.off[nl];
  T* minv = res + cells(0);
  T* adense = minv + S.n_coarse * S.n_coarse;
  T* scratch = adense + S.n_coarse * S.n_coarse;
  const int tid = threadIdx.x;
  for (int l = 0; l < nl; ++l) {
    const int n = cells(l), pad = S.lv[l].pad, na = n + pad;
    T* c = src(l) + n;
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
  // level l with its coefficients in shared memory
  const auto lv = [&](int l) {
    SubLevel<T> L = S.lv[l];
    const int n = L.nx * L.ny * L.nz, na = n + L.pad;
    const T* c = src(l) + n;
    L.cx = c;
    L.cy = c + na;
    L.cz = c + 2 * na;
    if (kSubIdiag<T>) L.id = c + 3 * na;
    return L;
  };
  // The set-up kernels that wrote the above are ordinary launches, complete
  // before any kernel of the cycle starts; what follows is the cycle's.
  pdl_wait();
#pragma unroll 4
  for (int q = tid; q < cells(0); q += kSubThreads) src(0)[q] = __ldcg(S.src_in + q);
  __syncthreads();
  for (int l = 0; l < nl - 1; ++l) {
    sub_sweeps(lv(l), sol(l), src(l), S.nu1, 0, true);
    sub_restrict(lv(l), sol(l), src(l), lv(l + 1), src(l + 1), res, S.nu1 > 0);
  }
  sub_coarse(S.n_coarse, minv, adense, src(nl - 1), sol(nl - 1), scratch);
  for (int l = nl - 2; l >= 0; --l) {
    sub_prolong(lv(l), sol(l), lv(l + 1), sol(l + 1), res, S.nu2 > 0 ? (S.reverse ? 0 : 1) : -1);
    sub_sweeps(lv(l), sol(l), src(l), S.nu2, S.reverse ? 1 : 0, false);
  }
  for (int q = tid; q < cells(0); q += kSubThreads) S.sol_out[q] = sol(0)[q];
}

template <typename T>
__global__ void __launch_bounds__(kSubThreads) k_subcycle(SubCycle<T> S) {
  pdl_launch();
  extern __shared__ unsigned char sub_raw[];
  subcycle_body(S, reinterpret_cast<T*>(sub_raw));
}

}  // namespace

template <typename T>
size_t subcycle_smem(const SubCycle<T>& S) {
  const int n0 = S.lv[0].nx * S.lv[0].ny * S.lv[0].nz;
  return (size_t)(S.off[S.nlev] + n0 + 2 * S.n_coarse * S.n_coarse + kMaxCoarse) * sizeof(T);
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
