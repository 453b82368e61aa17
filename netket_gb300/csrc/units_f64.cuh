// FP64 numbers as 64-bit integers in units of a power of two that a column of them
// shares: GB300 issues two FP64 operations per clock and SM against 128 integer ones.
#pragma once

#include "common.cuh"

namespace vmck {

typedef unsigned long long u64;

// Size of an entry for the largest of a column: the high word without its sign, its
// last bit set where only the low word is not 0.
__device__ __forceinline__ uint32_t size_word(double w) {
  return ((uint32_t)__double2hiint(w) & 0x7fffffffu) | (__double2loint(w) != 0 ? 1u : 0u);
}
// Whether entries below 2^(e - 1022) have the integer form
__device__ __forceinline__ bool exponent_fits(int e) { return e >= 200 && e <= 1900; }
// w, |w| < 2^(e - 1022), in units of unit_of(e, bits); |result| <= 2^bits
__device__ __forceinline__ long long to_units(double w, int e, int bits) {
  const int hi = __double2hiint(w), ew = (hi >> 20) & 0x7ff;
  const unsigned long long m =
      (unsigned long long)(uint32_t)((hi & 0xfffff) | (ew ? 0x100000 : 0)) << 32 |
      (uint32_t)__double2loint(w);
  const int s = bits - 53 - (e - (ew ? ew : 1));
  unsigned long long q = 0ull;
  if (s >= 0)
    q = m << s;
  else if (s > -55)
    q = (m + (1ull << (-s - 1))) >> -s;
  return hi < 0 ? -(long long)q : (long long)q;
}
__device__ __forceinline__ double unit_of(int e, int bits) {
  return __hiloint2double((e + 1 - bits) << 20, 0);
}
// bits that leave room for a sum of `terms` entries
__host__ __device__ __forceinline__ int sum_bits(int64_t terms) {
  int b = 62;
  while (terms > 1) {
    terms = (terms + 1) >> 1;
    --b;
  }
  return b;
}

// a + b, its rounding error added to low (infinities and NaN reach the sum alone)
__device__ __forceinline__ double two_sum(double a, double b, double &low) {
  const double s = a + b, v = s - a;
  const double e = (a - (s - v)) + (b - v);
  if (isfinite(s)) low += e;
  return s;
}

// a b / 2^64 for a, b <= 2^63; below = the 32 bits under it.  (The products that a
// 64-bit addend would carry into are written out: the compiler's own sequence takes
// twice the instructions.)
__device__ __forceinline__ unsigned long long mul_high(unsigned long long a, unsigned long long b,
                                                       uint32_t &below) {
  unsigned long long h;
  asm("{\n\t"
      ".reg .u32 al, ah, bl, bh, t, u, v;\n\t"
      ".reg .u64 m, w;\n\t"
      "mov.b64 {al, ah}, %2;\n\t"
      "mov.b64 {bl, bh}, %3;\n\t"
      "mul.hi.u32 t, al, bl;\n\t"
      "mov.b64 m, {t, 0};\n\t"
      "mad.wide.u32 m, al, bh, m;\n\t"
      "mad.wide.u32 m, ah, bl, m;\n\t"
      "mov.b64 {u, v}, m;\n\t"
      "mov.b64 w, {v, 0};\n\t"
      "mad.wide.u32 %0, ah, bh, w;\n\t"
      "mov.u32 %1, u;\n\t"
      "}"
      : "=l"(h), "=r"(below)
      : "l"(a), "l"(b));
  return h;
}

// 2^(-i / 32) in units of 2^-63
__device__ const u64 EXP2_NEG[32] = {
    0x8000000000000000ull, 0x7d41d96db915019dull, 0x7a92be8a92436616ull, 0x77f25ccdee6d7ae6ull,
    0x75606373ee921c97ull, 0x72dc8373be41a454ull, 0x70666f76154a7089ull, 0x6dfddbcbed791babull,
    0x6ba27e656b4eb57aull, 0x69540ec8f895722dull, 0x6712460a8fc24072ull, 0x64dcdec3371793d1ull,
    0x62b39508aa836d6full, 0x6096266533384a2bull, 0x5e8451cfac061b5full, 0x5c7dd7a3b17dcf75ull,
    0x5a827999fcef3242ull, 0x5891fac0e95612c8ull, 0x56ac1f752150a563ull, 0x54d0ad5a753e077cull,
    0x52ff6b54d8a89c75ull, 0x513821818624b40cull, 0x4f7a993048d088d7ull, 0x4dc69cdceaa72a9cull,
    0x4c1bf828c6dc54b8ull, 0x4a7a77d47f7b84b1ull, 0x48e1e9b9d588e19bull, 0x47521cc5a2e6a9e0ull,
    0x45cae0f1f545eb73ull, 0x444c0740496d4294ull, 0x42d561b3e6243d8aull, 0x4166c34c5615d0ecull,
};

// q = rho / (1 + rho), rho = e^(-2 theta), in units of 2^-63; all ones where theta is not
// finite.  With e = e^(-2 |theta|), r = 1 / (1 + e) is q (theta < 0) or 1 - q, so only
// absolute precision counts: e in fixed point (2 |theta| log2(e) = k + i / 32 + x / 32,
// a table for i and the Taylor series of 2^(-x / 32), whose terms from the fifth on fit
// in 32 bits), r by two Newton steps from a reciprocal in FP32.  Within 2^-58.8 of the
// exact value (rms 2^-60.5); FP64's exp and division take 64 us at 0.8 million values.
__device__ __forceinline__ u64 q_units(double theta) {
  const int hi = __double2hiint(theta), ew = (hi >> 20) & 0x7ff;
  if (ew == 0x7ff) return ~0ull;
  u64 r = 1ull << 63;
  if (fabs(theta) < 22.0) {  // else e < 2^-63
    const u64 m = (u64)(uint32_t)((hi & 0xfffff) | (ew ? 0x100000 : 0)) << 32 |
                  (uint32_t)__double2loint(theta);
    const int s = ew - 1017;  // |theta| in units of 2^-58
    const u64 a = s >= 0 ? m << s : s > -55 ? (m + (1ull << (-s - 1))) >> -s : 0ull;
    uint32_t below;
    const u64 h = mul_high(a, 0x5c551d94ae0bf85eull, below);  // 2 log2(e) 2^61
    const u64 y = h << 2 | below >> 30;                         // units of 2^-57
    const int k = (int)(y >> 57);
    const u64 table = EXP2_NEG[(int)(y >> 52) & 31];
    const u64 x = (y & ((1ull << 52) - 1)) << 11;
    const uint32_t xh = (uint32_t)(x >> 32);
    // v_n = (ln 2 / 16)^n / n! - v_(n+1) x / 2, in units of 2^-61
    uint32_t w = 710u;
    w = 131020u - __umulhi(w, xh);
    w = 21170451u - __umulhi(w, xh);
    w = 2932080444u - __umulhi(w, xh);
    u64 v = 338407833321ull - __umulhi(w, xh);
    v = 31246035387553ull - mul_high(v, x, below);
    v = 2163768014451044ull - mul_high(v, x, below);
    v = 99893036290645747ull - mul_high(v, x, below);
    v = 2305843009213693952ull - mul_high(v, x, below);
    const u64 d = (1ull << 60) + (mul_high(table, v, below) >> k);  // 1 + e
    // 1 / d in units of 2^-62
    const float seed = __fdividef(0x1p59f, __uint2float_rn((uint32_t)(d >> 32)));
    r = (u64)__float2uint_rn(seed) << 31;
    const long long e1 = (long long)((1ull << 58) - mul_high(d, r, below));
    r += ((long long)(r >> 31) * (e1 >> 8)) >> 19;
    const u64 g = mul_high(d, r, below);
    const long long e2 = (long long)((1ull << 61) - (g << 3 | below >> 29));
    r += ((long long)(r >> 31) * e2) >> 30;
    r = min(r << 1, 1ull << 63);
  }
  return hi >= 0 ? (1ull << 63) - r : r;
}

// Positive numbers m 2^e, 2^62 <= m < 2^63: products without the FP64 pipe
struct UFloat {
  u64 m;
  int e;
};
// f 2^e for 2^32 <= f < 2^63
__device__ __forceinline__ UFloat ufloat(u64 f, int e) {
  const int z = __clz((int)(f >> 32)) - 1;
  return {f << z, e - z};
}
__device__ __forceinline__ UFloat operator*(UFloat a, UFloat b) {
  uint32_t below;
  const u64 h = mul_high(a.m, b.m, below);  // 2^60 to 2^62
  const uint32_t lo = (uint32_t)h, hi = (uint32_t)(h >> 32);
  const int s = hi >> 29 ? 1 : 2;
  return {(u64)__funnelshift_l(lo, hi, s) << 32 | __funnelshift_l(below, lo, s),
          a.e + b.e + 64 - s};
}
__device__ __forceinline__ UFloat shfl_xor(UFloat a, int d) {
  return {__shfl_xor_sync(0xffffffffu, a.m, d), __shfl_xor_sync(0xffffffffu, a.e, d)};
}

}  // namespace vmck
