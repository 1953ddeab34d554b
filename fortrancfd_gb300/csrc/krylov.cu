// Vector kernels of the flexible GMRES outer iteration (sm_103a).
//
// Per Arnoldi step j, around the V-cycle on v_j:
//   k_gm_z       z_j = the V-cycle's result less its mean, into Z_j
//   k_apply_diag w = A z_j
//   k_gm_dots    the j+1 products V_i.w and w.w
//   k_gm_update  w -= sum_i h_i V_i, |w|^2 and 1/|w|
//   k_gm_next    v_{j+1} = w/|w| into V_{j+1} and into the V-cycle's right-hand side
// The products and the update are an FP64 operation per basis element each,
// for 8 bytes read: the FP64 pipe (2 lanes per clock and SM) takes 1.8 us per
// 1024^2 vector, memory 1.25 us, so both passes are bound by that pipe and
// everything beside the one operation is kept off it: w is read once for all
// vectors, and the sums of a warp are folded together (9 additions for eight
// sums, 40 one by one, which with four elements per thread were more than the
// products).  Both passes run twice in nearly every step: with a good preconditioner
// A M v is nearly v, and the first one takes most of w away (1024^2: 45 of 45 steps,
// 128^3: 15 of 15).  1024^2 in the stream of a step: products 26, 34 and 42 us with up
// to 7, 11 and 15 vectors, the update 48 on average, z 6, v 7, the mean 10; with a pass per
// vector, separate norms and two conversions 65 + 2 x 31 + 31 and two copies of 6.
// The sums keep a fixed order (thread: stride of the grid; warp: halves;
// block: warps in order; then blocks the same way), whatever is summed together.
// The basis is one array of vectors of n doubles
// at a stride of ld.
#include "gbmg_internal.h"
#include "idiv.h"
#include "pairs.cuh"
#include "pdl.cuh"

namespace gbmg {

namespace {

constexpr int kGmThreads = 256, kGmWarps = kGmThreads / 32;
constexpr int kGmVals = 32;  // sums of one launch
// Blocks of the products and of the update that are resident on an SM, and all
// that are launched: 1024 blocks took two to four rounds, the last one part empty
// (a step of 1024^2 343 us, now 317; of 64^3 196, now 174).
template <int G>
constexpr int kDotsBlocks = G <= 4 ? 3 : 2;
constexpr int kUpdateBlocks = 4;

// sums of the lanes' a[0..NV-1]: sum v in a[0] of the lanes v * 32/NV and up
template <int NV, int kOff = 16>
__device__ __forceinline__ void warp_fold(double* a) {
  if constexpr (NV > 1) {
    const bool up = threadIdx.x & kOff;
#pragma unroll
    for (int u = 0; u < NV / 2; ++u) {
      const double lo = a[u], hi = a[u + NV / 2];
      a[u] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, kOff);
    }
  } else {
    a[0] += __shfl_xor_sync(0xffffffffu, a[0], kOff);
  }
  if constexpr (kOff > 1) warp_fold<(NV > 1 ? NV / 2 : 1), kOff / 2>(a);
}

// sum of one value per thread of the block (valid in thread 0)
__device__ __forceinline__ double block_fold(double v, double* ws) {
  double a[1] = {v};
  warp_fold<1>(a);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = a[0];
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kGmWarps; ++w) t += ws[w];
  __syncthreads();
  return t;
}

// sum of the partials of a launch's blocks (valid in thread 0)
__device__ __forceinline__ double blocks_fold(const double* partials, int blocks, double* ws) {
  double a = 0.0;
  for (int b = threadIdx.x; b < blocks; b += kGmThreads) a += __ldcg(partials + b);
  return block_fold(a, ws);
}

// Whether a pass runs: the first one does, the second one where the first one's
// norms say so (the verdict is a double's bits: a comparison of its own in every
// thread, two roots, cost the FP64 pipe 20 us at 1024^2).
__device__ __forceinline__ bool gm_runs(const double* first) {
  return !first || __double_as_longlong(__ldcg(first + 2)) != 0;
}

// partials of V_i.w, i < cnt, and of w.w as the one after; 4 (G - 1) <= cnt < 4 G
template <int G>
__global__ void __launch_bounds__(kGmThreads, kDotsBlocks<G>)
    k_gm_dots(const double* __restrict__ V, size_t ld, int cnt, const double* __restrict__ w,
              size_t n, double* __restrict__ partials, const double* first) {
  pdl_enter();
  if (!gm_runs(first)) return;
  __shared__ double ws[kGmWarps][kGmVals];
  const size_t step = (size_t)gridDim.x * kGmThreads;
  double a[4 * G];
#pragma unroll
  for (int v = 0; v < 4 * G; ++v) a[v] = 0.0;
  // (the last group alone may be short, and holds w.w)
  const auto in = [&](int g, int u) { return g < G - 1 || u == 0 || 4 * g + u <= cnt; };
  const auto self = [&](int g, int u) { return g == G - 1 && 4 * g + u == cnt; };
  size_t q = (size_t)blockIdx.x * kGmThreads + threadIdx.x;
  for (; q + step < n; q += 2 * step) {
    const double w0 = w[q], w1 = w[q + step];
    const double* v = V + q;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      double v0[4], v1[4];
#pragma unroll
      for (int u = 0; u < 4; ++u, v += ld)
        if (in(g, u)) {
          const double* p = self(g, u) ? w + q : v;
          v0[u] = p[0];
          v1[u] = p[step];
        }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (in(g, u)) {
          a[4 * g + u] += v0[u] * w0;
          a[4 * g + u] += v1[u] * w1;
        }
    }
  }
  if (q < n) {
    const double w0 = w[q];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (in(g, u)) a[4 * g + u] += (self(g, u) ? w : V + (size_t)(4 * g + u) * ld)[q] * w0;
  }
  const int lane = threadIdx.x & 31;
  double* mine = ws[threadIdx.x >> 5];
#pragma unroll
  for (int g = 0; g + 1 < G; g += 2) {
    warp_fold<8>(a + 4 * g);
    if (lane % 4 == 0) mine[4 * g + lane / 4] = a[4 * g];
  }
  if constexpr (G & 1) {
    warp_fold<4>(a + 4 * (G - 1));
    if (lane % 8 == 0) mine[4 * (G - 1) + lane / 8] = a[4 * (G - 1)];
  }
  __syncthreads();
  if ((int)threadIdx.x <= cnt) {
    double t = 0.0;
#pragma unroll
    for (int u = 0; u < kGmWarps; ++u) t += ws[u][threadIdx.x];
    partials[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
}

// out[i] = the sum of the blocks' partials, a block per sum
__global__ void __launch_bounds__(kGmThreads) k_gm_finish(const double* __restrict__ partials,
                                                          int blocks, double* __restrict__ out,
                                                          const double* first) {
  pdl_enter();
  if (!gm_runs(first)) return;
  __shared__ double ws[kGmWarps];
  const double t = blocks_fold(partials + (size_t)blockIdx.x * blocks, blocks, ws);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// w += sign * sum_i coef[i] V_i (added in index order); kNorm: nrm[0] = |w|^2,
// nrm[1] = 1/|w| (0 for w = 0), and from the first pass nrm[2] = 1 when it left less
// than 0.7 of the length sqrt(*before) ("twice is enough"): a second pass that is
// not needed takes the first one's norms
template <bool kNorm>
__global__ void __launch_bounds__(kGmThreads, kUpdateBlocks)
    k_gm_update(double* __restrict__ w, const double* __restrict__ V, size_t ld,
                const double* __restrict__ coef, int cnt, double sign, size_t n, double* partials,
                unsigned int* counter, double* nrm, const double* before, const double* first) {
  pdl_enter();
  if (!gm_runs(first)) {
    if (kNorm && blockIdx.x == 0 && threadIdx.x < 2) nrm[threadIdx.x] = first[threadIdx.x];
    return;
  }
  __shared__ double ws[kGmWarps], c[kGmVals];
  __shared__ bool last;
  if (threadIdx.x < (unsigned)cnt) c[threadIdx.x] = coef[threadIdx.x];
  __syncthreads();
  const size_t step = (size_t)gridDim.x * kGmThreads;
  double s = 0.0;
  size_t q = (size_t)blockIdx.x * kGmThreads + threadIdx.x;
  for (; q + step < n; q += 2 * step) {
    const double w0 = w[q], w1 = w[q + step];
    double a0 = 0.0, a1 = 0.0;
    const double* v = V + q;
#pragma unroll 4
    for (int i = 0; i < cnt; ++i, v += ld) {
      a0 += c[i] * v[0];
      a1 += c[i] * v[step];
    }
    const double x0 = w0 + sign * a0, x1 = w1 + sign * a1;
    w[q] = x0;
    w[q + step] = x1;
    if (kNorm) {
      s += x0 * x0;
      s += x1 * x1;
    }
  }
  if (q < n) {
    double a = 0.0;
    for (int i = 0; i < cnt; ++i) a += c[i] * V[(size_t)i * ld + q];
    const double x = w[q] + sign * a;
    w[q] = x;
    if (kNorm) s += x * x;
  }
  if (kNorm) {
    const double t = block_fold(s, ws);
    if (threadIdx.x == 0) {
      partials[blockIdx.x] = t;
      __threadfence();
      last = atomicAdd(counter, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const double r = blocks_fold(partials, (int)gridDim.x, ws);
    if (threadIdx.x == 0) {
      nrm[0] = r;
      nrm[1] = r > 0.0 ? 1.0 / sqrt(r) : 0.0;
      if (before) nrm[2] = sqrt(r) < 0.7 * sqrt(*before) ? 1.0 : 0.0;
      *counter = 0u;
    }
  }
}

// v = scale * w (scale read from inv when there is one), and v as the V-cycle's
// right-hand side: src64 (K = kZ64), or rounded to float in the level's layout.
// w may be src64.
template <int K>
__global__ void __launch_bounds__(kGmThreads)
    k_gm_next(double* __restrict__ v, const double* w, const double* __restrict__ inv, double scale,
              double* src64, float* __restrict__ src32, size_t n, PairRows P, size_t hstride) {
  const double a = inv ? *inv : scale;
  const size_t step = (size_t)gridDim.x * kGmThreads;
  for (size_t m = (size_t)blockIdx.x * kGmThreads + threadIdx.x; m < n / 2; m += step) {
    const double2 x = reinterpret_cast<const double2*>(w)[m];
    const double2 y = make_double2(a * x.x, a * x.y);
    reinterpret_cast<double2*>(v)[m] = y;
    if constexpr (K == kZ64) reinterpret_cast<double2*>(src64)[m] = y;
    else store_pair32<K>(src32, m, y.x, y.y, P, hstride);
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
    const double y = a * w[n - 1];
    v[n - 1] = y;
    if constexpr (K == kZ64) src64[n - 1] = y;
    else src32[n - 1] = (float)y;
  }
}

// The sum of the V-cycle's FP32 result into R.result[slot], the additions of k_sum on
// its FP64 copy: kSumTogether of its blocks in one, their warps folded together
// (1024^2: 18.7 us before, beside the copy)
constexpr int kSumTogether = 4;

template <int K>
__global__ void __launch_bounds__(kGmThreads)
    k_gm_sum(const float* __restrict__ z, size_t n, PairRows P, size_t hstride, int blocks,
             ReduceScratch R, int slot) {
  static_assert(kGmThreads == kRedThreads, "k_sum's blocks");
  __shared__ double ws[kGmWarps][kSumTogether], fin[kGmWarps];
  __shared__ bool last;
  const size_t step = (size_t)blocks * kGmThreads;
  const int b0 = blockIdx.x * kSumTogether;
  double a[kSumTogether] = {0.0, 0.0, 0.0, 0.0};
  const auto load = [&](size_t q) {
    if constexpr (K == kZSplit)
      return z[(size_t)(pair_colour(P, q >> 1) ^ (int)(q & 1)) * hstride + (q >> 1)];
    else return z[q];
  };
  size_t q = (size_t)b0 * kGmThreads + threadIdx.x;
  for (; q < n; q += step) {
    float v[kSumTogether];
#pragma unroll
    for (int u = 0; u < kSumTogether; ++u) {
      const size_t e = q + (size_t)u * kGmThreads;
      v[u] = b0 + u < blocks && e < n ? load(e) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kSumTogether; ++u)
      if (b0 + u < blocks && q + (size_t)u * kGmThreads < n) a[u] += float_to_double_int(v[u]);
  }
  const int lane = threadIdx.x & 31;
  warp_fold<kSumTogether>(a);
  if (lane % (32 / kSumTogether) == 0) ws[threadIdx.x >> 5][lane / (32 / kSumTogether)] = a[0];
  __syncthreads();
  if (threadIdx.x < kSumTogether) {
    const int u = threadIdx.x;
    const double t = ((ws[0][u] + ws[4][u]) + (ws[2][u] + ws[6][u])) +
                     ((ws[1][u] + ws[5][u]) + (ws[3][u] + ws[7][u]));
    if (b0 + u < blocks) R.partials[b0 + u] = t;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(R.counter, 1u) == gridDim.x - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  double acc[1] = {0.0};
  for (int b = threadIdx.x; b < blocks; b += kGmThreads) acc[0] += __ldcg(&R.partials[b]);
  warp_fold<1>(acc);
  if (lane == 0) fin[threadIdx.x >> 5] = acc[0];
  __syncthreads();
  if (threadIdx.x == 0) {
    R.result[slot] = ((fin[0] + fin[4]) + (fin[2] + fin[6])) + ((fin[1] + fin[5]) + (fin[3] + fin[7]));
    *R.counter = 0u;
  }
}

// out = z - (sum of z)/n
template <int K>
__global__ void __launch_bounds__(kGmThreads)
    k_gm_z(const void* __restrict__ z, double* __restrict__ out, size_t n, PairRows P,
           size_t hstride, const double* __restrict__ sum) {
  const double mean = div_int(*sum, rcp_int((double)n));
  const size_t step = (size_t)gridDim.x * kGmThreads;
  for (size_t m = (size_t)blockIdx.x * kGmThreads + threadIdx.x; m < n / 2; m += step) {
    const double2 x = widen(load_pair<K>(z, m, P, hstride));
    reinterpret_cast<double2*>(out)[m] = make_double2(x.x - mean, x.y - mean);
  }
  if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) out[n - 1] = load_one<K>(z, n - 1) - mean;
}

unsigned gm_blocks(size_t items, unsigned most) {
  const size_t b = (items + kGmThreads - 1) / kGmThreads;
  return (unsigned)std::max<size_t>(1, std::min<size_t>(b, most));
}

}  // namespace

namespace {
// (returns the number of blocks)
template <int G>
int dots_groups(cudaStream_t s, const double* V, size_t ld, int cnt, const double* w, size_t n,
                double* partials, const double* first) {
  if constexpr (G > 1)
    if (cnt < 4 * (G - 1)) return dots_groups<G - 1>(s, V, ld, cnt, w, n, partials, first);
  const unsigned b = gm_blocks(n, 152 * kDotsBlocks<G>);
  launch_pdl(k_gm_dots<G>, dim3(b), dim3(kGmThreads), 0, s, V, ld, cnt, w, n, partials, first);
  return (int)b;
}
}  // namespace

void launch_gm_dots(cudaStream_t s, const double* V, size_t ld, int cnt, const double* w, size_t n,
                    double* partials, double* out, const double* first) {
  static_assert(kGmresRestart < kGmVals, "sums of one launch");
  const int b = dots_groups<kGmVals / 4>(s, V, ld, cnt, w, n, partials, first);
  launch_pdl(k_gm_finish, dim3((unsigned)cnt + 1u), dim3(kGmThreads), 0, s,
             (const double*)partials, b, out, first);
}

void launch_gm_update(cudaStream_t s, double* w, const double* V, size_t ld, const double* coef,
                      int cnt, double sign, size_t n, double* partials, unsigned int* counter,
                      double* nrm, const double* before, const double* first) {
  static_assert(152 * kUpdateBlocks <= kGmresBlocks && 152 * kDotsBlocks<1> <= kGmresBlocks,
                "partials");
  const dim3 b(gm_blocks(n, 152 * kUpdateBlocks)), t(kGmThreads);
  if (nrm)
    launch_pdl(k_gm_update<true>, b, t, 0, s, w, V, ld, coef, cnt, sign, n, partials, counter, nrm, before, first);
  else
    launch_pdl(k_gm_update<false>, b, t, 0, s, w, V, ld, coef, cnt, sign, n, partials, counter, nrm, before, first);
}

void launch_gm_sum(cudaStream_t s, const PcgVec& z, const ReduceScratch& R, int slot) {
  if (z.z64) return launch_sum(s, z.z64, z.n, R, slot);
  const PairRows P = pair_rows(z.nx, z.ny);
  const int blocks = sum_blocks(z.n, R);
  const unsigned b = (unsigned)(blocks + kSumTogether - 1) / kSumTogether;
  if (z.hstride) k_gm_sum<kZSplit><<<b, kGmThreads, 0, s>>>(z.z32, z.n, P, z.hstride, blocks, R, slot);
  else k_gm_sum<kZ32><<<b, kGmThreads, 0, s>>>(z.z32, z.n, P, 0, blocks, R, slot);
}

void launch_gm_next(cudaStream_t s, double* v, const double* w, const double* inv, double scale,
                    double* src64, float* src32, const PcgVec& z) {
  const PairRows P = pair_rows(z.nx, z.ny);
  const unsigned b = gm_blocks(z.n / 2, 152 * 8);
  if (src64) k_gm_next<kZ64><<<b, kGmThreads, 0, s>>>(v, w, inv, scale, src64, src32, z.n, P, 0);
  else if (z.hstride)
    k_gm_next<kZSplit><<<b, kGmThreads, 0, s>>>(v, w, inv, scale, src64, src32, z.n, P, z.hstride);
  else k_gm_next<kZ32><<<b, kGmThreads, 0, s>>>(v, w, inv, scale, src64, src32, z.n, P, 0);
}

void launch_gm_z(cudaStream_t s, const PcgVec& z, double* out, const double* sum) {
  const PairRows P = pair_rows(z.nx, z.ny);
  const unsigned b = gm_blocks(z.n / 2, 152 * 8);
  if (z.z64) k_gm_z<kZ64><<<b, kGmThreads, 0, s>>>(z.z64, out, z.n, P, 0, sum);
  else if (z.hstride) k_gm_z<kZSplit><<<b, kGmThreads, 0, s>>>(z.z32, out, z.n, P, z.hstride, sum);
  else k_gm_z<kZ32><<<b, kGmThreads, 0, s>>>(z.z32, out, z.n, P, 0, sum);
}

}  // namespace gbmg
