// Pairs of cells (2m, 2m+1) of a V-cycle's result, for the vector passes of the
// Krylov iterations: FP64, FP32, or FP32 in the colour-split layout (cell q in
// half (i+j+k)&1 at q/2; a pair shares a row, nx being even there).
#pragma once

#include <algorithm>

#include "dword.cuh"
#include "gbmg_internal.h"
#include "reduce.cuh"

namespace gbmg {

enum : int { kZ64 = 0, kZ32 = 1, kZSplit = 2 };

// row and plane of a pair by products with 2^64/divisor (an integer division
// by a variable goes through the FP64 pipe): exact for m * divisor < 2^64
struct PairRows {
  unsigned hx, ny;
  unsigned long long rx, ry;  // floor(2^64 / hx) + 1, floor(2^64 / ny) + 1; 0 for a divisor of 1
};

__device__ __forceinline__ unsigned long long div_by(unsigned long long m, unsigned long long r) {
  return r ? __umul64hi(m, r) : m;
}

__device__ __forceinline__ int pair_colour(const PairRows& P, unsigned long long m) {
  const unsigned long long row = div_by(m, P.rx);
  const unsigned long long k = div_by(row, P.ry);
  return (int)((row - k * P.ny + k) & 1ull);  // (j + k) & 1: the colour of cell 2m
}

// cells 2m and 2m+1 of z as floats
template <int K>
__device__ __forceinline__ float2 load_pair32(const float* __restrict__ z, size_t m,
                                              const PairRows& P, size_t hstride) {
  if constexpr (K == kZSplit) {
    const int c = pair_colour(P, m);
    return make_float2(z[(size_t)c * hstride + m], z[(size_t)(1 - c) * hstride + m]);
  } else {
    return reinterpret_cast<const float2*>(z)[m];
  }
}

template <int K>
__device__ __forceinline__ auto load_pair(const void* __restrict__ z, size_t m, const PairRows& P,
                                          size_t hstride) {
  if constexpr (K == kZ64) return reinterpret_cast<const double2*>(z)[m];
  else return load_pair32<K>(static_cast<const float*>(z), m, P, hstride);
}

__device__ __forceinline__ double2 widen(double2 v) { return v; }
__device__ __forceinline__ double2 widen(float2 v) {
  return make_double2(float_to_double_int(v.x), float_to_double_int(v.y));
}

// a last cell without a partner (n odd; never split)
template <int K>
__device__ __forceinline__ double load_one(const void* __restrict__ z, size_t q) {
  if constexpr (K == kZ64) return static_cast<const double*>(z)[q];
  else return (double)static_cast<const float*>(z)[q];
}

// cells 2m and 2m+1 rounded to float, K = kZ32 or kZSplit
template <int K>
__device__ __forceinline__ void store_pair32(float* out, size_t m, double a, double b,
                                             const PairRows& P, size_t hstride) {
  const float fa = dw_from_double_int(a).hi, fb = dw_from_double_int(b).hi;
  if constexpr (K == kZSplit) {
    const int c = pair_colour(P, m);
    out[(size_t)c * hstride + m] = fa;
    out[(size_t)(1 - c) * hstride + m] = fb;
  } else {
    reinterpret_cast<float2*>(out)[m] = make_float2(fa, fb);
  }
}

// the factor of div_by for a divisor
inline unsigned long long div_rcp(int d) { return d == 1 ? 0ull : ~0ull / (unsigned)d + 1; }

inline PairRows pair_rows(int nx, int ny) {
  PairRows P{};
  P.hx = (unsigned)std::max(nx / 2, 1);
  P.ny = (unsigned)ny;
  P.rx = div_rcp((int)P.hx);
  P.ry = div_rcp(ny);
  return P;
}

inline unsigned blocks_of(size_t items, const ReduceScratch& R) {
  const size_t b = (items + kRedThreads - 1) / kRedThreads;
  return (unsigned)std::max<size_t>(
      1, std::min<size_t>(b, std::min<size_t>(152 * 8, (size_t)R.max_blocks)));
}

}  // namespace gbmg
