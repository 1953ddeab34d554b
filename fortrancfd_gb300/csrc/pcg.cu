// Vector passes of the flexible-CG outer iteration (sm_103a).
//
// One iteration on the finest level is z = M r (a V-cycle), then
//   k_pcg_sum        the sum of z (its mean is projected out)
//   k_pcg_dots       z - mean into z_old, with r.z and r.z_old before it
//   k_pcg_direction  d = z + beta d, beta = (r.z - r.z_old)/(r.z of the last)
//   k_apply_diag     q = A d and d.q
//   k_pcg_step       p += alpha d, r -= alpha q, |r|^2, and r rounded to float
//                    for the next FP32 V-cycle
// The residual follows the recursion; the solve loop restates it as b - A p in
// FP64 every few iterations and before it accepts a solution.  On small grids and
// near the accuracy that FP64 allows it is recomputed every iteration (k_pcg_x,
// then the residual kernel).
// Recomputing it always, with one pass per vector operation, read and wrote
// 208 bytes and issued 37 FP64 operations per cell and iteration: 10.6 of the 13.7
// ms of a 512^3 iteration.  These passes move 156 bytes with 15 operations (mixed;
// FP64 160 with 16; the FP64 pipe runs 2 lanes per clock and SM, so an operation
// per cell costs as much as 11 bytes); with b - A p in place of the recursion 188 with
// 28 (FP64 184 with 29).
// z is read straight from the V-cycle's result: FP64, FP32, or FP32 in the
// colour-split layout (cell q in half (i+j+k)&1 at q/2).  All passes work on
// pairs of cells (2m, 2m+1), which share a row when nx is even.
#include "dword.cuh"
#include "gbmg_internal.h"
#include "pairs.cuh"
#include "reduce.cuh"

namespace gbmg {

namespace {

// sum of floats in three cascaded parts (TwoSum at each step; Ogita, Rump and
// Oishi, "Accurate sum and dot product", SIAM J. Sci. Comput. 26(6), 2005):
// rounds at 2^-72, below an FP64 sum, on the FP32 pipes
struct FloatSum {
  float hi = 0.f, mid = 0.f, lo = 0.f;
  __device__ __forceinline__ void add(float x) {
    const dw a = two_sum(hi, x);
    hi = a.hi;
    const dw b = two_sum(mid, a.lo);
    mid = b.hi;
    lo += b.lo;
  }
  __device__ __forceinline__ double value() const { return (double)hi + ((double)mid + (double)lo); }
};

template <int K>
__global__ void __launch_bounds__(kRedThreads) k_pcg_sum(const void* __restrict__ z, size_t n,
                                                         PairRows P, size_t hstride,
                                                         ReduceScratch R, int slot) {
  double acc[1] = {0.0};
  if constexpr (K == kZ64) {
    stride4(n, [&](size_t q) { return static_cast<const double*>(z)[q]; },
            [&](size_t, double v) { acc[0] += v; });
  } else {
    // (the cells in the same order for both layouts)
    FloatSum s;
    const float* f = static_cast<const float*>(z);
    stride4(n / 2, [&](size_t m) { return load_pair32<K>(f, m, P, hstride); },
            [&](size_t, float2 v) {
              s.add(v.x);
              s.add(v.y);
            });
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) s.add(f[n - 1]);
    acc[0] = s.value();
  }
  grid_sum_finish<1>(acc, R, slot);
}

template <int K>
__global__ void __launch_bounds__(kRedThreads)
    k_pcg_dots(const void* __restrict__ z, const double* __restrict__ r, double* zold, size_t n,
               PairRows P, size_t hstride, ReduceScratch R) {
  const double mean = R.result[kSlotSum] / (double)n;
  double acc[2] = {0.0, 0.0};
  double2* zo = reinterpret_cast<double2*>(zold);
  const double2* r2 = reinterpret_cast<const double2*>(r);
  const auto one = [&](size_t m, double2 z2, double2 rv, double2 o) {
    const double a = z2.x - mean, b = z2.y - mean;
    zo[m] = make_double2(a, b);
    acc[0] += rv.x * a;
    acc[0] += rv.y * b;
    acc[1] += rv.x * o.x;
    acc[1] += rv.y * o.y;
  };
  // two pairs in flight per thread (four took 114 registers and ran at half
  // the rate: 212 us at 256^3)
  const size_t step = (size_t)gridDim.x * blockDim.x, pairs = n / 2;
  size_t m = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; m + step < pairs; m += 2 * step) {
    const auto za = load_pair<K>(z, m, P, hstride);
    const auto zb = load_pair<K>(z, m + step, P, hstride);
    const double2 ra = r2[m], oa = zo[m], rb = r2[m + step], ob = zo[m + step];
    one(m, widen(za), ra, oa);
    one(m + step, widen(zb), rb, ob);
  }
  if (m < pairs) one(m, widen(load_pair<K>(z, m, P, hstride)), r2[m], zo[m]);
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const size_t q = n - 1;
    const double a = load_one<K>(z, q) - mean, o = zold[q];
    zold[q] = a;
    acc[0] += r[q] * a;
    acc[1] += r[q] * o;
  }
  grid_sum_finish<2>(acc, R, kSlotDot);
}

__global__ void __launch_bounds__(kRedThreads)
    k_pcg_direction(double* d, const double* __restrict__ z, size_t n, ReduceScratch R,
                    int first) {
  const double beta =
      first ? 0.0 : (R.result[kSlotDot] - R.result[kSlotDot + 1]) / R.result[kSlotDot2 + 1];
  stride4(n, [&](size_t q) { return make_double2(z[q], first ? 0.0 : d[q]); },
          [&](size_t q, double2 v) { d[q] = first ? v.x : v.x + beta * v.y; });
}

__global__ void __launch_bounds__(kRedThreads)
    k_pcg_x(double* x, const double* __restrict__ d, size_t n, ReduceScratch R) {
  const double alpha = R.result[kSlotDot] / R.result[kSlotDot2];
  stride4(n, [&](size_t q) { return make_double2(x[q], d[q]); },
          [&](size_t q, double2 v) { x[q] = v.x + alpha * v.y; });
}

// r32 (K = kZ32, kZSplit): the new residual rounded to float.  n is even: an odd grid
// has no coarser level and at most kMaxCoarse cells, too few for the recursion.
template <int K>
__global__ void __launch_bounds__(kRedThreads)
    k_pcg_step(double* x, const double* __restrict__ d, double* r, const double* __restrict__ q,
               float* r32, size_t n, PairRows P, size_t hstride, ReduceScratch R) {
  const double alpha = R.result[kSlotDot] / R.result[kSlotDot2];
  double acc[1] = {0.0};
  double2* x2 = reinterpret_cast<double2*>(x);
  double2* r2 = reinterpret_cast<double2*>(r);
  const double2* d2 = reinterpret_cast<const double2*>(d);
  const double2* q2 = reinterpret_cast<const double2*>(q);
  const size_t step = (size_t)gridDim.x * blockDim.x;
  const auto one = [&](size_t m, double2 xv, double2 dv, double2 rv, double2 qv) {
    x2[m] = make_double2(xv.x + alpha * dv.x, xv.y + alpha * dv.y);
    const double a = rv.x - alpha * qv.x, b = rv.y - alpha * qv.y;
    r2[m] = make_double2(a, b);
    acc[0] += a * a;
    acc[0] += b * b;
    if constexpr (K != kZ64) store_pair32<K>(r32, m, a, b, P, hstride);
  };
  size_t m = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t pairs = n / 2;
  for (; m + step < pairs; m += 2 * step) {
    const double2 xa = x2[m], da = d2[m], ra = r2[m], qa = q2[m];
    const double2 xb = x2[m + step], db = d2[m + step], rb = r2[m + step], qb = q2[m + step];
    one(m, xa, da, ra, qa);
    one(m + step, xb, db, rb, qb);
  }
  if (m < pairs) one(m, x2[m], d2[m], r2[m], q2[m]);
  grid_sum_finish<1>(acc, R, kSlotNorm);
}

}  // namespace

void launch_pcg_sum(cudaStream_t s, const PcgVec& v, const ReduceScratch& R, int slot) {
  const PairRows P = pair_rows(v.nx, v.ny);
  // 16 cells a thread: the FP64 additions that join the threads' sums cost as
  // much as reading 50 cells each (1024^2: 14.8 us at 4 cells a thread)
  const unsigned b = std::max(blocks_of(v.n / 16, R), std::min(blocks_of(v.n, R), 152u));
  if (v.z64) k_pcg_sum<kZ64><<<b, kRedThreads, 0, s>>>(v.z64, v.n, P, 0, R, slot);
  else if (v.hstride) k_pcg_sum<kZSplit><<<b, kRedThreads, 0, s>>>(v.z32, v.n, P, v.hstride, R, slot);
  else k_pcg_sum<kZ32><<<b, kRedThreads, 0, s>>>(v.z32, v.n, P, 0, R, slot);
}

void launch_pcg_dots(cudaStream_t s, const PcgVec& v, const double* r, double* zold,
                     const ReduceScratch& R) {
  const PairRows P = pair_rows(v.nx, v.ny);
  const unsigned b = blocks_of(v.n / 2, R);
  if (v.z64) k_pcg_dots<kZ64><<<b, kRedThreads, 0, s>>>(v.z64, r, zold, v.n, P, 0, R);
  else if (v.hstride) k_pcg_dots<kZSplit><<<b, kRedThreads, 0, s>>>(v.z32, r, zold, v.n, P, v.hstride, R);
  else k_pcg_dots<kZ32><<<b, kRedThreads, 0, s>>>(v.z32, r, zold, v.n, P, 0, R);
}

void launch_pcg_direction(cudaStream_t s, double* d, const double* z, size_t n,
                          const ReduceScratch& R, int first) {
  const size_t b = (n + kRedThreads - 1) / kRedThreads;
  k_pcg_direction<<<(unsigned)std::max<size_t>(1, std::min<size_t>(b, 152 * 16)), kRedThreads, 0,
                    s>>>(d, z, n, R, first);
}

void launch_pcg_x(cudaStream_t s, double* x, const double* d, size_t n, const ReduceScratch& R) {
  k_pcg_x<<<blocks_of(n, R), kRedThreads, 0, s>>>(x, d, n, R);
}

void launch_pcg_step(cudaStream_t s, double* x, const double* d, double* r, const double* q,
                     float* r32, const PcgVec& v, const ReduceScratch& R) {
  const PairRows P = pair_rows(v.nx, v.ny);
  const unsigned b = blocks_of(v.n / 2, R);
  if (!r32) k_pcg_step<kZ64><<<b, kRedThreads, 0, s>>>(x, d, r, q, r32, v.n, P, 0, R);
  else if (v.hstride) k_pcg_step<kZSplit><<<b, kRedThreads, 0, s>>>(x, d, r, q, r32, v.n, P, v.hstride, R);
  else k_pcg_step<kZ32><<<b, kRedThreads, 0, s>>>(x, d, r, q, r32, v.n, P, 0, R);
}

}  // namespace gbmg
