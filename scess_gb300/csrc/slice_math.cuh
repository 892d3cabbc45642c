// Digit extraction and recombination of the sliced FP64 GEMM, usable on host and
// device (the host form is what the CPU test exercises).
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

namespace scess {

#ifdef __CUDACC__
#define SCESS_HD __host__ __device__ __forceinline__
#else
#define SCESS_HD inline
#endif

SCESS_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
SCESS_HD double double_of(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
SCESS_HD int clz32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}
// Upper word of (hi, lo) << n, 0 <= n <= 31.
SCESS_HD uint32_t funnel_l(uint32_t hi, uint32_t lo, int n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, n);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << n) >> 32);
#endif
}
SCESS_HD int rint_i32(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)std::nearbyintf(x);
#endif
}

// Fixed-point value of a finite x relative to a row whose largest biased
// exponent is emax >= x's: F = x 2^(60 - E), E = emax - 1022, |F| <= 2^60,
// rounded to nearest (exact while x is within 2^-7 of the row's largest).
SCESS_HD int64_t slice_fixed(double x, int emax) {
  const uint64_t b = bits_of(x);
  int be = (int)((b >> 52) & 0x7ff);
  uint64_t m = b & 0xfffffffffffffull;
  if (be) m |= 1ull << 52;
  else be = 1;  // subnormal (or zero): no implicit bit
  if (emax < 1) emax = 1;
  const int sh = emax - be - 7;
  int64_t F;
  if (sh <= 0) F = (int64_t)(m << (-sh));
  else if (sh < 62) F = (int64_t)((m + (1ull << (sh - 1))) >> sh);
  else F = 0;
  return (b >> 63) ? -F : F;
}

// |x| relative to its row's largest exponent as BF16 bits, rounded down: |x| 2^(1022 - emax), at least
// 2^-60 unless x is zero.
SCESS_HD uint32_t slice_magnitude(double x, int emax) {
  const uint64_t b = bits_of(x) & 0x7fffffffffffffffull;
  const int be = (int)(b >> 52), gap = emax - be;
  if (b == 0) return 0u;
  return be == 0 || gap > 59 ? (127 - 60) << 7 : (uint32_t)(126 - gap) << 7 | ((uint32_t)(b >> 45) & 0x7fu);
}

// F + kDigitBias has digit p (p = 1 .. 6) in bits [9 (6 - p), 9 (6 - p) + 9)
// offset by 256, and digit 0 above bit 54.
constexpr int64_t kDigitBias = 256ll * (1ll + (1ll << 9) + (1ll << 18) + (1ll << 27) + (1ll << 36) +
                                        (1ll << 45));
SCESS_HD int slice_digit(int64_t G, int p) {
  return p == 0 ? (int)(G >> 54) : (int)((G >> (9 * (6 - p))) & 511) - 256;
}

// 2^n as a double, n clamped to the representable powers.
SCESS_HD double power_of_two(int n) {
  n = n < -1074 ? -1074 : (n > 1023 ? 1023 : n);
  return double_of(n < -1022 ? 1ull << (n + 1074) : (uint64_t)(n + 1023) << 52);
}

// (T + w 2^-fs) 2^sc rounded to FP64 (|T| < 2^62, 1 <= fs <= 31, -900 <= sc <= 800),
// its sign bit xor-ed by flip unless it is zero.
SCESS_HD double slice_value_plain(int64_t T, int w, int fs, int sc, uint32_t flip) {
  const uint64_t H = (uint64_t)(T + (int64_t)(w >> fs));
  const uint32_t f = (uint32_t)w << (32 - fs);
  const uint32_t sgn = (uint32_t)((int64_t)H >> 63);
  const uint32_t h1 = (uint32_t)(H >> 32) ^ sgn, h0 = (uint32_t)H ^ sgn, l = f ^ sgn;
  // The leading nonzero word first: (a, b, c) of (h1, h0, l).  The magnitude of a negative sum is
  // its complement and one more in the last place, which is the complement with ones without end:
  // they follow l, and the rounding carries them up.
  const bool m1 = h1 == 0u, m2 = m1 && h0 == 0u;
  const uint32_t a = m2 ? l : (m1 ? h0 : h1), b = m2 ? sgn : (m1 ? l : h0), c = m1 ? sgn : l;
  const int lz = clz32(a);
  const uint32_t x1 = funnel_l(a, b, lz & 31), x0 = funnel_l(b, c, lz & 31);
  const int be = sc + 1023 + 63 - lz - (m1 ? 32 : 0) - (m2 ? 32 : 0);
  // 53 bits of (x1, x0), the half bit rounded up; the carry runs into the exponent
  const uint64_t mant = ((((uint64_t)x1 << 32) | x0) >> 11) + ((x0 >> 10) & 1u);
  const double v = double_of(((uint64_t)(((uint32_t)(be - 1) << 20) + ((sgn & 0x80000000u) ^ flip)) << 32) + mant);
  return a == 0u ? 0.0 : v;
}
// The same for any sc.
SCESS_HD double slice_value(int64_t T, int w, int fs, int sc, uint32_t flip) {
  const int scc = sc < -900 ? -900 : (sc > 800 ? 800 : sc);
  double v = slice_value_plain(T, w, fs, scc, flip);
  // beyond the normal numbers: one more rounding, to the place or to infinity
  if (sc < scc) v = v * power_of_two(-100) * power_of_two(sc - scc + 100);
  else if (sc > scc) v *= power_of_two(sc - scc);
  return v;
}

}  // namespace scess
