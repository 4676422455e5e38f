// FP64 arithmetic of the elementwise kernels in integer instructions, with the
// bits that the IEEE operation gives.
//
// GB300's FP64 unit takes about half a lane per cycle and SM in these kernels (nine
// sums a particle kept it 73 % busy for 29 us at 400k particles): a warp's FP64
// operation costs the issue slots of ~200 other instructions. The products, conversions
// and comparisons below take 10 to 30, the sums ~60. A few sums are left to the unit,
// which then works beside them. Operands outside the common range (zero, subnormal,
// infinite, NaN, a result outside the normal range) take the plain operation.
//
// Host and device code alike: the functions are compared with the host's own
// arithmetic in the CPU tests.
#pragma once

#include <stdint.h>

#include <cstring>

#ifdef __CUDACC__
#define IDPD_HD __host__ __device__ __forceinline__
#else
#define IDPD_HD inline
#endif

namespace idpd {

IDPD_HD uint64_t f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
IDPD_HD double f64_from(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
// The operations of the rare operands; volatile, so that they are not computed ahead of
// the test that asks for them.
IDPD_HD double plain_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  double c;
  asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(c) : "d"(a), "d"(b));
  return c;
#else
  return a * b;
#endif
}
IDPD_HD double plain_add(double a, double b) {
#ifdef __CUDA_ARCH__
  double c;
  asm volatile("add.rn.f64 %0, %1, %2;" : "=d"(c) : "d"(a), "d"(b));
  return c;
#else
  return a + b;
#endif
}
IDPD_HD float plain_f32(double a) {
#ifdef __CUDA_ARCH__
  float c;
  asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(c) : "d"(a));
  return c;
#else
  return (float)a;
#endif
}
IDPD_HD int plain_int(double a) {
#ifdef __CUDA_ARCH__
  int c;
  asm volatile("cvt.rzi.s32.f64 %0, %1;" : "=r"(c) : "d"(a));
  return c;
#else
  return (int)a;
#endif
}
IDPD_HD double plain_f64(int n) {
#ifdef __CUDA_ARCH__
  double c;
  asm volatile("cvt.rn.f64.s32 %0, %1;" : "=d"(c) : "r"(n));
  return c;
#else
  return (double)n;
#endif
}
IDPD_HD int clz64(uint64_t x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}

constexpr uint64_t kMant = 0xFFFFFFFFFFFFFull, kHidden = 0x10000000000000ull;

// a * b rounded to nearest even, for a factor b used many times (the integer path: b > 0 and
// normal).
IDPD_HD double mul_f64(double a, double b) {
  const uint64_t ab = f64_bits(a), bb = f64_bits(b);
  // a factor that is zero, subnormal, not finite or negative gets an exponent that no product
  // takes (once for all its uses)
  constexpr int kNoFactor = 8192;
  const int fb = (int)(bb >> 52), eb = (uint32_t)(fb - 1) > 2045u ? kNoFactor : fb;
  const int ea = (int)(ab >> 52) & 0x7ff;
  int e = ea + eb - 1022;
  if (ea == 0 || ea == 0x7ff || e < 2 || e > 2045) {
    if ((ab << 1) == 0 && eb != kNoFactor) return a;  // a zero keeps its sign
    return plain_mul(a, b);
  }
  const uint64_t m = (ab & kMant) | kHidden, f = (bb & kMant) << 11 | 0x8000000000000000ull;
  // the 117-bit product m f = hi 2^64 + lo, hi in [2^51, 2^53)
  const uint32_t m0 = (uint32_t)m, m1 = (uint32_t)(m >> 32);
  const uint32_t f0 = (uint32_t)f, f1 = (uint32_t)(f >> 32);
  const uint64_t p00 = (uint64_t)m0 * f0;
  const uint64_t p01 = (uint64_t)m0 * f1 + (p00 >> 32);
  const uint64_t p10 = (uint64_t)m1 * f0 + (uint32_t)p01;
  uint64_t hi = (uint64_t)m1 * f1 + (p01 >> 32) + (p10 >> 32);
  uint64_t lo = p10 << 32 | (uint32_t)p00;
  if (!(hi >> 52)) {
    hi = hi << 1 | lo >> 63;
    lo <<= 1;
    e -= 1;
  }
  hi += (lo >> 63) & (uint64_t)(((lo << 1) != 0) | (hi & 1));
  return f64_from((ab & 0x8000000000000000ull) | (((uint64_t)(uint32_t)(e - 1) << 52) + hi));
}

// a + b rounded to nearest even.
IDPD_HD double add_f64(double a, double b) {
  uint64_t x = f64_bits(a), y = f64_bits(b);
  if ((x << 1) < (y << 1)) {  // |x| >= |y|
    const uint64_t t = x;
    x = y;
    y = t;
  }
  const int ex = (int)(x >> 52) & 0x7ff, ey = (int)(y >> 52) & 0x7ff;
  if (ey == 0 || ex < 128 || ex > 0x7fd) {
    if ((y << 1) == 0 && (x << 1) != 0) return f64_from(x);
    return plain_add(a, b);
  }
  // ten bits below the last place; the smaller operand's bits beyond them as one sticky bit
  const uint64_t mx = ((x & kMant) | kHidden) << 10, my = ((y & kMant) | kHidden) << 10;
  const int d = ex - ey;
  uint64_t t = d < 64 ? my >> d : 0;
  t |= (uint64_t)(d >= 64 || (t << d) != my);
  const uint64_t s = (x ^ y) >> 63 ? mx - t : mx + t;
  if (s == 0) return 0.0;
  const int lz = clz64(s);
  const uint64_t q = s << lz;
  const uint64_t r = q & 0x7ff;
  uint64_t m = q >> 11;
  m += (uint64_t)(r > 0x400) | (uint64_t)(r == 0x400 && (m & 1));
  return f64_from((x & 0x8000000000000000ull) | (((uint64_t)(uint32_t)(ex - lz) << 52) + m));
}

// n * b rounded to nearest even, n >= 0, b > 0 normal.
IDPD_HD double mul_int_f64(int n, double b) {
  if (n == 0) return 0.0;
  if (n >= 2048) return plain_mul(plain_f64(n), b);
  const uint64_t bb = f64_bits(b);
  const uint64_t p = ((bb & kMant) | kHidden) * (uint64_t)(uint32_t)n;  // below 2^64
  const int lz = clz64(p);
  const uint64_t q = p << lz;
  const uint64_t r = q & 0x7ff;
  uint64_t m = q >> 11;
  m += (uint64_t)(r > 0x400) | (uint64_t)(r == 0x400 && (m & 1));
  return f64_from(((uint64_t)((int)(bb >> 52) + 10 - lz) << 52) + m);
}

// q 2^-26 for |q| < 2^51 (exact).
IDPD_HD double scale_force(long long q) {
  const uint64_t a = q < 0 ? 0ull - (uint64_t)q : (uint64_t)q;
  if (a == 0) return 0.0;
  const int lz = clz64(a);
  const uint64_t m = a << (lz - 11);  // hidden bit at bit 52; lz >= 13
  return f64_from((q < 0 ? 0x8000000000000000ull : 0ull) |
                  (((uint64_t)(1059 - lz) << 52) + m));
}

// (float)x, rounded to nearest even.
IDPD_HD float to_f32(double x) {
  const uint64_t b = f64_bits(x);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ff;
  if (e - 897u > 252u) return plain_f32(x);  // not a normal float
  const uint64_t r = b + 0xFFFFFFFull + ((b >> 29) & 1);
  const uint32_t f = ((uint32_t)(r >> 29) - (896u << 23)) | ((uint32_t)(b >> 32) & 0x80000000u);
#ifdef __CUDA_ARCH__
  return __uint_as_float(f);
#else
  float y;
  std::memcpy(&y, &f, 4);
  return y;
#endif
}

// (int)x truncated, for x >= 0 below 2^31 (0 for negative zero and below 1).
IDPD_HD int to_int(double x) {
  const uint64_t b = f64_bits(x);
  const int e = ((int)(b >> 52) & 0x7ff) - 1023;
  if (e < 0) return 0;
  if (e > 30) return plain_int(x);
  return (int)(((b & kMant) | kHidden) >> (52 - e));
}

// The cell of coordinate x on an axis of nc cells, inv_cs cells per unit length: the
// truncated product, and the nearest cell for a coordinate outside the box, 0 for NaN (a run
// that diverged, a caller's rows that are refused later), so that the result is always an
// index below nc.
IDPD_HD int cell_index(double x, double inv_cs, int nc) {
  const double q = mul_f64(x, inv_cs);
  const uint64_t b = f64_bits(q);
  if (b >= 0x41E0000000000000ull)  // 2^31 and above, infinite, NaN, negative
    return b <= 0x7FF0000000000000ull ? nc - 1 : 0;
  const int c = to_int(q);
  return c >= nc ? nc - 1 : c;
}

// |x| > y for y >= 0, x finite.
IDPD_HD bool abs_above(double x, double y) { return (f64_bits(x) << 1) > (f64_bits(y) << 1); }

// x in units of 2^-32, truncated towards zero; |x| < 2^20 (in_fix).
IDPD_HD bool in_fix(double x) { return ((int)(f64_bits(x) >> 52) & 0x7ff) < 1043; }
IDPD_HD long long to_fix(double x) {
  const uint64_t b = f64_bits(x);
  const int sh = 1043 - ((int)(b >> 52) & 0x7ff);
  const uint64_t m = sh > 63 ? 0 : ((b & kMant) | kHidden) >> sh;
  return (long long)b < 0 ? -(long long)m : (long long)m;
}

}  // namespace idpd
