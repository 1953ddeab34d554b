// Correctly rounded FP64 quotients and products in integer and FP32 arithmetic.
//
// GB300's FP64 pipe takes one warp instruction per 16 cycles of an SM (2 lanes
// per clock), so a kernel that keeps the reference's divisions to reproduce
// its doubles is bound by that pipe while the integer and FP32 pipes idle (a
// quotient is about 30 instructions here, a product about 22, at one to two
// warp instructions per cycle).  These use none of it:
//
//   rcp_int(b)     64-bit fixed-point reciprocal of b's significand: a float
//                  reciprocal, one step of residual correction in float (about
//                  44 bits) and one Newton step in 64-bit integers (62 bits);
//   div_int(a, r)  the quotient's bits by a 64 x 64 -> 64 high product, then
//                  the rounding decided by the sign of the exact remainder
//                  against the midpoint, so the result is RN(a/b) for every
//                  input, as IEEE division gives it;
//   div_3(a, s)    RN(a / (3 2^s)): the quotient by 3 is at least 1/6 ulp from
//                  every midpoint, so the high product alone decides.
//
//   mul_int(a, b)  RN(a b) from the high half of the significands' product (the
//                  low half is formed only when the high one ends in a tie);
//   mul_k<K>(a)    RN(K a) for a small whole number K;
//   sqrt_int(a)    RN(sqrt(a)).
//
// One rcp_int serves all quotients with its divisor.  Subnormal, infinite or
// NaN operands and results near the ends of the exponent range take the
// ordinary operation.  Plain C++ for the host too (the CPU test sweeps it
// against the host's division, with the float reciprocal displaced by its
// error bound).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define GB_HD __host__ __device__ __forceinline__
#else
#define GB_HD inline
#endif

namespace gbmg {

GB_HD uint64_t idiv_bits(double x) {
#if defined(__CUDA_ARCH__)
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return u;
#endif
}

GB_HD double idiv_double(uint64_t u) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}

GB_HD float idiv_float(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float x;
  std::memcpy(&x, &u, 4);
  return x;
#endif
}

GB_HD uint32_t idiv_fbits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return u;
#endif
}

GB_HD uint64_t idiv_mulhi(uint64_t a, uint64_t b) {
#if defined(__CUDA_ARCH__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

// a float within 2^-23 (relative) of 1/x, x in [1, 2)
#if !defined(__CUDA_ARCH__)
inline int& idiv_seed_shift() {  // host tests: displace the seed by this many ulps
  static int s = 0;
  return s;
}
#endif
GB_HD float idiv_seed(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  float r = 1.0f / x;
  return x == 1.0f ? r : idiv_float(idiv_fbits(r) + (uint32_t)idiv_seed_shift());
#endif
}

GB_HD float idiv_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}

// The ordinary division as a call: inlined, its FP64 instructions would be
// issued for every element.
#if defined(__CUDACC__)
__host__ __device__ __noinline__ inline double idiv_ieee(double a, double b) { return a / b; }
#else
inline double idiv_ieee(double a, double b) { return a / b; }
#endif

GB_HD double idiv_mul64(double a, double b) {
#if defined(__CUDA_ARCH__)
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}

GB_HD double idiv_fma64(double a, double b, double c) {
#if defined(__CUDA_ARCH__)
  return __fma_rn(a, b, c);
#else
  return __builtin_fma(a, b, c);
#endif
}

struct RcpInt {
  uint64_t y;   // 2^127 / (significand << 11), within 4 units below
  uint64_t m;   // significand (53 bits)
  double b;
  int e;        // biased exponent; 0 when b is outside the fast range
};

GB_HD RcpInt rcp_int(double b) {
  const uint64_t u = idiv_bits(b);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  RcpInt r;
  r.b = b;
  r.m = (u & 0xfffffffffffffull) | (1ull << 52);
  // positive and normal
  const uint32_t e = hi >> 20;
  r.e = (e - 1u) < 2046u ? (int)e : 0;
  // significand = x + t 2^-23 + (below 2^-46), x in [1, 2), t in [0, 1)
  const float x = idiv_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29));
  const float t = idiv_float(0x3f800000u | ((lo >> 6) & 0x7fffffu)) - 1.0f;
  float y0 = idiv_seed(x);
  y0 = y0 > 0.5f ? y0 : 0.5f;
  float d = idiv_fma(-x, y0, 1.0f);
  d = idiv_fma(t, y0 * -0x1p-23f, d);
  const float c = y0 * idiv_fma(d, d, d);  // 1/significand - y0, to 2^-45
  const int ci = (int)idiv_fbits(idiv_fma(c, 0x1p44f, 12582912.0f)) - 0x4B400000;
  // y0 2^24 is an integer in [2^23, 2^24]; 3 units of 2^-44 below keep y an
  // underestimate
  const uint32_t yi = idiv_fbits(y0) - 0x3f000000u + 0x800000u;
  const uint64_t y = ((uint64_t)yi << 40) + (uint64_t)((int64_t)(ci - 3) << 20);
  // Newton: 2^127 - (m << 11) y = (dd - [0, 1)) 2^64
  const uint64_t dd = (1ull << 63) - idiv_mulhi(r.m << 11, y);
  r.y = y + (((uint64_t)(uint32_t)(y >> 32) * (uint32_t)(dd - 1)) >> 31);
  return r;
}

// RN(a / b) for r = rcp_int(b)
GB_HD double div_int(double a, const RcpInt& r) {
  const uint64_t u = idiv_bits(a);
  const int ea = (int)((u >> 52) & 0x7ff);
  const int e = ea - r.e + 1022;  // biased exponent of the result, less one
  if ((unsigned)(ea - 1) >= 2046u || r.e == 0 || (unsigned)(e - 2) >= 2040u)
    return (u << 1) == 0 && r.e != 0 ? a : idiv_ieee(a, r.b);  // (a zero over b > 0 is itself)
  const uint64_t ma = (u & 0xfffffffffffffull) | (1ull << 52);
  // q = floor-ish (a/b significands) 2^63, at most 5 units low
  const uint64_t q = idiv_mulhi(ma << 11, r.y);
  const int big = (int)(q >> 63);
  const uint64_t k = q >> (10 + big);
  // a/b against the midpoint (2k+1)/2: the sign of the exact difference
  const int64_t rest = (int64_t)((ma << (54 - big)) - r.m * (2 * k + 1));
  const uint64_t v = ((uint64_t)(uint32_t)(e - 1 + big) << 52) + k + (rest > 0 ? 1u : 0u);
  return idiv_double(v | (u & 0x8000000000000000ull));
}

// RN(a / (3 2^s)), s in 0..2
GB_HD double div_3(double a, int s) {
  const uint64_t u = idiv_bits(a);
  const int ea = (int)((u >> 52) & 0x7ff);
  if ((unsigned)(ea - 8) >= 2039u) return (u << 1) ? idiv_ieee(a, (double)(3 << s)) : a;
  const uint64_t ma = (u & 0xfffffffffffffull) | (1ull << 52);
  const uint64_t q = idiv_mulhi(ma << 11, 0xaaaaaaaaaaaaaaaaull);  // 2^65/3
  const int big = (int)(q >> 63);
  const uint64_t k = (q + (512ull << big)) >> (10 + big);
  const uint64_t v = ((uint64_t)(uint32_t)(ea - 3 - s + big) << 52) + k;
  return idiv_double(v | (u & 0x8000000000000000ull));
}

#if defined(__CUDACC__)
__host__ __device__ __noinline__ inline double imul_ieee(double a, double b) { return a * b; }
#else
inline double imul_ieee(double a, double b) { return a * b; }
#endif

// RN(a b)
GB_HD double mul_int(double a, double b) {
  const uint64_t u = idiv_bits(a), w = idiv_bits(b);
  const int ea = (int)((u >> 52) & 0x7ff), eb = (int)((w >> 52) & 0x7ff);
  const int e = ea + eb - 1023;
  if ((unsigned)(ea - 1) >= 2046u || (unsigned)(eb - 1) >= 2046u || (unsigned)(e - 2) >= 2040u) {
    // (a zero times a finite value is a zero)
    if (((u << 1) == 0 || (w << 1) == 0) && ea < 2047 && eb < 2047)
      return idiv_double((u ^ w) & 0x8000000000000000ull);
    return imul_ieee(a, b);
  }
  const uint64_t ma = ((u & 0xfffffffffffffull) | (1ull << 52)) << 11;
  const uint64_t mb = ((w & 0xfffffffffffffull) | (1ull << 52)) << 11;
  const uint64_t q = idiv_mulhi(ma, mb);
  const int big = (int)(q >> 63);
  const int sh = 10 + big;
  const uint64_t half = 512ull << big;
  uint64_t k = (q + half) >> sh;
  // the kept high part ends in exactly one half: a tie only if the low part is 0
  if ((((uint32_t)q ^ (uint32_t)half) & ((2u << (sh - 1)) - 1u)) == 0 && ma * mb == 0) k &= ~1ull;
  const uint64_t v = ((uint64_t)(uint32_t)(e - 1 + big) << 52) + k;
  return idiv_double(v | ((u ^ w) & 0x8000000000000000ull));
}

// RN(K a), 3 <= K <= 15
template <int K>
GB_HD double mul_k(double a) {
  static_assert(K >= 3 && K <= 15, "K");
  constexpr int B = K >= 8 ? 3 : (K >= 4 ? 2 : 1);  // 2^B <= K
  const uint64_t u = idiv_bits(a);
  const int ea = (int)((u >> 52) & 0x7ff);
  if ((unsigned)(ea - 1) >= 2040u) return (u << 1) == 0 ? a : imul_ieee(a, (double)K);
  const uint64_t v = ((u & 0xfffffffffffffull) | (1ull << 52)) * (uint64_t)K;
  const int big = (int)(v >> (53 + B));
  const int sh = B + big;
  const uint64_t k = (v + (((1u << sh) >> 1) - 1u) + ((v >> sh) & 1u)) >> sh;
  const uint64_t r = ((uint64_t)(uint32_t)(ea - 1 + sh) << 52) + k;
  return idiv_double(r | (u & 0x8000000000000000ull));
}

// x 2^K by the exponent
template <int K>
GB_HD double scale2(double x) {
  const uint64_t u = idiv_bits(x);
  if ((unsigned)((int)((u >> 52) & 0x7ff) - 64) < 1900u)
    return idiv_double(u + ((uint64_t)(int64_t)K << 52));
  return (u << 1) == 0 ? x : imul_ieee(x, K < 0 ? 1.0 / (double)(1ll << -K) : (double)(1ll << K));
}

#if defined(__CUDACC__)
__host__ __device__ __noinline__ inline double isqrt_ieee(double a) { return sqrt(a); }
#else
inline double isqrt_ieee(double a) { return std::sqrt(a); }
#endif

// a float within 2^-22.9 (relative) of x^-1/2, x in [1, 4)
GB_HD float isqrt_seed(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  const float r = (float)(1.0 / std::sqrt((double)x));
  return x == 1.0f ? r : idiv_float(idiv_fbits(r) + (uint32_t)idiv_seed_shift());
#endif
}

// RN(sqrt(a)): a float square root, two steps s += (x - s^2)/(2 s) with exact
// integer remainders (44 bits, then all), the last bit by the sign of
// N - (K + 1/2)^2.
GB_HD double sqrt_int(double a) {
  const uint64_t u = idiv_bits(a);
  const uint32_t ea = (uint32_t)(u >> 52);
  if (ea - 1u >= 2046u) return isqrt_ieee(a);  // not positive, normal and finite
  const int odd = (int)(~ea & 1u);  // odd exponent (the bias is odd)
  const uint64_t m = ((u & 0xfffffffffffffull) | (1ull << 52)) << odd;  // x 2^52, x in [1, 4)
  const float x = idiv_float((odd ? 0x40000000u : 0x3f800000u) | (uint32_t)((u >> 29) & 0x7fffffu));
  const float r = isqrt_seed(x);
  // r 2^31 and s0 2^31 (s0 = x r in [1, 2)) as integers
  const uint32_t ri = (idiv_fbits(r) - 0x3f000000u + 0x800000u) << 7;
  float s0 = x * r;
  s0 = s0 < 1.0f ? 1.0f : (s0 > 1.9999999f ? 1.9999999f : s0);
  const uint32_t si = ((idiv_fbits(s0) & 0x7fffffu) | 0x800000u) << 8;
  const int64_t d0 = (int64_t)((m << 10) - (uint64_t)si * si);  // (x - s0^2) 2^62
  const int64_t s1 = (int64_t)((uint64_t)si << 31) + (((int64_t)(int32_t)(d0 >> 13) * ri) >> 19);
  const uint64_t h = (uint64_t)s1 >> 11;  // s 2^51
  const int64_t d1 = (int64_t)((m << 50) - h * h);  // x 2^102 - h^2
  uint64_t k = 2 * h + (uint64_t)(((int64_t)(int32_t)(d1 >> 31) * ri) >> 51);  // s 2^52, N = x 2^104
  const int64_t d2 = (int64_t)((m << 52) - k * k);
  k += (d2 > (int64_t)k ? 1u : 0u) - (uint64_t)(d2 <= -(int64_t)k ? 1u : 0u);
  const uint32_t e = (ea + 1023u - (uint32_t)odd) >> 1;  // exponent of the root
  return idiv_double(((uint64_t)(e - 1) << 52) + k);
}

// exponent field in place: larger for larger magnitudes, infinities and NaN on top
GB_HD uint32_t idiv_mag(double x) { return (uint32_t)(idiv_bits(x) >> 32) & 0x7ff00000u; }
constexpr uint32_t kMagOk = (1023u + 900u) << 20;  // below: |x| < 2^900

// Bits of a magnitude slightly above ls_wid (1 - 1e-12): |phi| beyond it gives
// |RN(phi/ls_wid)| > 1 - 1e-12, the clipping threshold of ls_funs, whatever the
// rounding (margin 1e-15).
inline long long ls_outside_bits(double ls_wid) {
  return (long long)idiv_bits(ls_wid * (1.0 - 1e-12) * (1.0 + 1e-15));
}

// whether |b| lies in 2^-60..2^60, so that quotients of ordinary values by it stay
// in the normal range
inline bool divisor_ok(double b) {
  const double m = b < 0 ? -b : b;
  return m >= 0x1p-60 && m <= 0x1p60;
}

// ---- division by a constant known on the host --------------------------------
// kDivExact: h is a power of two, x / h adds to the exponent.
// kDivPair:  x / h = fma(x, y, x yl) with y + yl = 1/h to 106 bits, two FP64
//            operations (N. Brisebarre, J.-M. Muller, S. K. Raina,
//            "Accelerating Correctly Rounded Floating-Point Division when the
//            Divisor Is Known in Advance", IEEE Trans. Computers 53(8), 2004).
//            The sum before its rounding errs by at most 2^-52 ulp, so it can
//            only go wrong for an x whose quotient lies that close to a
//            midpoint; const_div finds all such x (at most a few, from a
//            linear congruence) and tests them.
// kDivKnown: some such x fails (or h is negative): with y = 1/h rounded to nearest,
//            q0 = x y is within two ulps of the quotient, one correction by the
//            remainder, q1 = q0 + (x - h q0) y, brings it within one, and a second
//            one rounds correctly (P. Markstein, "Computation of elementary
//            functions on the IBM RISC System/6000 processor", IBM J. Res. Dev.
//            34(1), 1990): five operations.
// kDivIeee:  h out of range: the division itself.
enum : int { kDivIeee = 0, kDivExact = 1, kDivPair = 2, kDivKnown = 3 };

struct ConstDiv {
  double h, y, yl;
  int mode;
  int ex;  // kDivExact: log2 of 1/h
  RcpInt r;
};

GB_HD double div_const(const ConstDiv& c, double x) {
  // |x| in 2^-900 .. 2^900: nothing underflows or overflows
  const uint64_t u = idiv_bits(x);
  if ((unsigned)((int)((u >> 52) & 0x7ff) - 123) < 1800u) {
    if (c.mode == kDivExact) return idiv_double(u + ((uint64_t)(int64_t)c.ex << 52));
    if (c.mode == kDivPair) return idiv_fma64(x, c.y, idiv_mul64(x, c.yl));
    if (c.mode == kDivKnown) {
      const double q0 = idiv_mul64(x, c.y);
      const double q1 = idiv_fma64(idiv_fma64(-c.h, q0, x), c.y, q0);
      return idiv_fma64(idiv_fma64(-c.h, q1, x), c.y, q1);
    }
  }
  // (a zero is its own quotient when h > 0)
  return (u << 1) == 0 && (c.mode == kDivPair || c.mode == kDivExact) ? x : idiv_ieee(x, c.h);
}

// the same quotient on the integer pipes (kernels bound by the FP64 pipe: about
// 30 instructions at one to two a cycle, against two at 16 cycles each)
GB_HD double div_const_i(const ConstDiv& c, double x) {
  const uint64_t u = idiv_bits(x);
  if (c.mode == kDivExact && (unsigned)((int)((u >> 52) & 0x7ff) - 123) < 1800u)
    return idiv_double(u + ((uint64_t)(int64_t)c.ex << 52));
  return div_int(x, c.r);
}

// the constant for div_const_i alone (without const_div's search, about a
// microsecond of the host)
inline ConstDiv const_div_i(double h) {
  ConstDiv c{h, 1.0 / h, 0.0, kDivIeee, 0, rcp_int(h)};
  int ex;
  if (h >= 0x1p-60 && h <= 0x1p60 && std::frexp(h, &ex) == 0.5) {
    c.mode = kDivExact;
    c.ex = 1 - ex;
  }
  return c;
}

inline ConstDiv const_div(double h) {
  ConstDiv c = const_div_i(h);
  if (c.mode == kDivExact || !divisor_ok(h)) return c;
  int ex;
  c.mode = kDivKnown;
  if (!(h > 0)) return c;
  c.yl = std::fma(-h, c.y, 1.0) / h;
  // x = A 2^i, h = B 2^j with 53-bit A and B; A 2^s - B m = delta for the odd
  // m of a midpoint, s = 53 (A >= B) or 54 (A < B), within 2^-52 ulp of it
  // when |delta| <= 4.  With B = 2^t Bo: delta = 2^t delta', and A is fixed
  // modulo Bo.
  const uint64_t B = (uint64_t)std::ldexp(std::frexp(h, &ex), 53);
  uint64_t Bo = B;
  int t = 0;
  while (!(Bo & 1)) { Bo >>= 1; ++t; }
  if (t > 2) { c.mode = kDivPair; return c; }
  bool ok = true;
  for (int s = 53; s <= 54; ++s) {
    // inverse of 2^(s-t) modulo Bo by halving
    uint64_t inv = 1;
    for (int i = 0; i < s - t; ++i) inv = (inv & 1) ? (inv >> 1) + (Bo >> 1) + 1 : inv >> 1;
    for (int64_t d = -4; d <= 4; ++d) {
      if (d == 0 || (d & ((1 << t) - 1))) continue;
      const int64_t dp = d / (1 << t);
      const uint64_t mag = (uint64_t)(dp < 0 ? -dp : dp);
      uint64_t A = (uint64_t)((unsigned __int128)mag * inv % Bo);
      if (dp < 0 && A) A = Bo - A;
      for (; A < (1ull << 53); A += Bo) {
        if (A < (1ull << 52)) continue;
        const double x = (double)A, b = (double)B;
        const double y = 1.0 / b, yl = std::fma(-b, y, 1.0) / b;
        if (std::fma(x, y, x * yl) != x / b) ok = false;
      }
    }
  }
  if (ok) c.mode = kDivPair;
  return c;
}

}  // namespace gbmg
