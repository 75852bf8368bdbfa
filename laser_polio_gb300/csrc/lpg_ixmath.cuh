/*
 * lpg_ixmath.cuh — exp2, exp and log1p to double precision with 64-bit
 * integer arithmetic.
 *
 * A GB300 SM issues about two FP64 operations per clock and 128 integer or
 * FP32 ones, so a 64 x 64-bit high product (eight instructions) costs an
 * eighth of one FP64 multiplication.  The functions here work on fixed-point
 * fractions with 63 or 64 bits, good to about 2^-60, and round to a double
 * once: they are as accurate as the FP64 library's and several times
 * cheaper.  Methods: table reductions (Tang) and short Taylor series.
 * Tables are formed on the host in long double (ix_tables).
 */
#ifndef LPG_IXMATH_CUH
#define LPG_IXMATH_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

#define IX_EXP_N 128
#define IX_LOG_N 128
struct IxTables {
  uint64_t exp2_t[IX_EXP_N];  /* 2^(j/128), 63 fraction bits */
  uint64_t log_c[IX_LOG_N];   /* c_j near 1/(1 + (j + 1/2)/128), a multiple of 2^-10, 63 fraction bits */
  uint64_t log_v[IX_LOG_N];   /* -ln c_j, 63 fraction bits */
};

#define IX_LN2_64 0xB17217F7D1CF79ACULL   /* ln 2, 64 fraction bits */
#define IX_LOG2E_63 0xB8AA3B295C17F0BCULL /* 1/ln 2, 63 fraction bits */

/* m 2^(n - 63) as a double, m with its top bit set, -1022 <= n <= 1022. */
__device__ __forceinline__ double ix_double(uint64_t m, int n) {
  const uint64_t r = (m >> 11) + ((m >> 10) & 1);
  return __longlong_as_double((long long)(((uint64_t)(int64_t)(n + 1022) << 52) + r));
}

/* 2^(f 2^-64), 63 fraction bits (the top bit set). */
__device__ __forceinline__ uint64_t ix_exp2_frac(const IxTables* T, uint64_t f) {
  const uint64_t t = T->exp2_t[f >> 57];
  const uint64_t z = __umul64hi(f & ((1ULL << 57) - 1), IX_LN2_64); /* < 2^-7.5 */
  const uint64_t z2 = __umul64hi(z, z);
  /* e^z - 1 = z + z^2 (1/2 + z (1/6 + z (1/24 + z (1/120 + z/720)))) */
  const uint32_t zs = (uint32_t)(z >> 25); /* 39 fraction bits */
  const uint32_t d = 0x02222222u + (__umulhi(zs, 0x005b05b0u) >> 7);
  const uint32_t a = 0x0aaaaaabu + (__umulhi(zs, d) >> 7);
  const uint64_t b = 0x2aaaaaaaaaaaaaabULL + ((uint64_t)zs * a >> 7);
  const uint64_t c = (1ULL << 63) + __umul64hi(z, b);
  return t + __umul64hi(t, z + __umul64hi(z2, c)) + 2; /* 2: the mean of what the products cut off */
}

/* |x| as an integer with 53 fraction bits, |x| < 2^10. */
__device__ __forceinline__ uint64_t ix_fixed53(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int ex = (int)(b >> 52 & 0x7ff);
  const uint64_t m = (b & 0xfffffffffffffULL) | (ex ? 1ULL << 52 : 0);
  const int sh = 1022 - ex; /* m 2^(ex - 1075 + 53) */
  return sh <= 0 ? m << -sh : sh > 60 ? 0 : (m + (1ULL << (sh - 1))) >> sh;
}

/* 0 <= x < hi (hi > 0) by the bits: a comparison of doubles is an FP64
 * operation.  False for -0 and NaN. */
__device__ __forceinline__ bool ix_below(double x, double hi) {
  return (uint64_t)__double_as_longlong(x) < (uint64_t)__double_as_longlong(hi);
}

/* Quotients by one divisor d: where d lies in [1, 2^500) the hardware's
 * estimate of 1/d, one Newton step and Markstein's correction (P. Markstein,
 * "Computation of elementary functions on the IBM RISC System/6000
 * processor", IBM J. Res. Develop. 34, 1990): the quotient, its remainder by
 * a fused multiply-add, and that times 1/d added.  The estimate's 20 bits
 * become 76, so the quotient is the correctly rounded one but for one in
 * millions, in five FP64 operations, three for a further dividend. */
struct IxDivisor {
  double d, y;
  bool fast;
  __device__ __forceinline__ explicit IxDivisor(double d_) : d(d_) {
    const uint32_t e = (uint32_t)((uint64_t)__double_as_longlong(d) >> 52); /* sign and exponent */
    fast = e - 1023u < 500u;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    y = __fma_rn(y, __fma_rn(-d, y, 1.0), y);
  }
  /* n / d */
  __device__ __forceinline__ double of(double n) const {
    const uint64_t b = (uint64_t)__double_as_longlong(n) << 1;
    if (!fast || ((uint32_t)(b >> 53) - 523u >= 1000u && b != 0)) return n / d;
    const double q = n * y;
    return __fma_rn(__fma_rn(-q, d, n), y, q);
  }
};

/* e^-x for 0 <= x < 2^-7: 1 - d, d = x - x^2 (1/2 - x (1/6 - x (1/24 - x
 * (1/120 - x (1/720 - x/5040))))) with 71 fraction bits, so that the result
 * is the correctly rounded one but for about one x in 1e5 at 2^-10 (1 - e^-x
 * of a small rate, which the expected exposures sum, shows its last bit). */
__device__ __forceinline__ double ix_exp_neg_small(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int sh = 1004 - (int)(b >> 52); /* x 2^71 = m 2^(ex - 1004) */
  const uint64_t m = (b & 0xfffffffffffffULL) | 1ULL << 52;
  const uint64_t X = sh <= 0 ? m << -sh : sh > 60 ? 0 : m >> sh;
  const uint64_t x2 = __umul64hi(X, X);   /* 78 fraction bits */
  const uint32_t xs = (uint32_t)(X >> 32); /* 39 */
  const uint32_t e = 0x005b05b0u - (__umulhi(xs, 0x000d00d0u) >> 7);
  const uint32_t d = 0x02222222u - (__umulhi(xs, e) >> 7);
  const uint32_t a = 0x0aaaaaabu - (__umulhi(xs, d) >> 7);
  const uint64_t c6 = 0x2aaaaaaaaaaaaaabULL - ((uint64_t)xs * a >> 7);
  const uint64_t c2 = (1ULL << 63) - (__umul64hi(X, c6) >> 7);
  const uint64_t D = X - (__umul64hi(x2, c2) >> 7);
  return __longlong_as_double((long long)((1021ULL << 52) + (1ULL << 53) - ((D + (1ULL << 17)) >> 18)));
}

/* e^-x for 0 <= x < 700, from x / ln 2 with 64 fraction bits. */
__device__ __forceinline__ double ix_exp_neg(const IxTables* T, double x) {
  if (ix_below(x, 0x1p-7)) return ix_exp_neg_small(x);
  int n;
  uint64_t f;
  if (ix_below(x, 0.5)) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int sh = 1012 - (int)(b >> 52 & 0x7ff); /* x 2^63 = m 2^(ex - 1012) */
    const uint64_t m = (b & 0xfffffffffffffULL) | 1ULL << 52;
    const uint64_t X = sh <= 0 ? m << -sh : sh > 60 ? 0 : m >> sh;
    f = 0ULL - (__umul64hi(X, IX_LOG2E_63) << 2 | X * IX_LOG2E_63 >> 62);
    n = f ? -1 : 0;
  } else {
    const uint64_t X = ix_fixed53(x); /* exact: x has no lower bits */
    const uint64_t hi = __umul64hi(X, IX_LOG2E_63), lo = X * IX_LOG2E_63; /* x / ln 2, 52 and 64 fraction bits */
    f = 0ULL - (hi << 12 | lo >> 52);
    n = -(int)(hi >> 52) - (f ? 1 : 0);
  }
  return ix_double(ix_exp2_frac(T, f), n);
}

/* v 2^-63 as a double. */
__device__ __forceinline__ double ix_frac_double(uint64_t v) {
  if (v == 0) return 0.0;
  const int lz = __clzll((long long)v);
  return ix_double(v << lz, -lz);
}

/* ln(1 + y) for 2^-5 <= y < 2^60: 1 + y = 2^e m, r = m c_j - 1. */
__device__ __forceinline__ double ix_log1p(const IxTables* T, double y) {
  const uint64_t b = (uint64_t)__double_as_longlong(y);
  const int ex = (int)(b >> 52) - 1023; /* -5 .. 59 */
  const uint64_t f = ((b & 0xfffffffffffffULL) | 1ULL << 52) << 11; /* y = f 2^(ex - 63) */
  uint64_t m;
  int e;
  if (ex < 0) {
    m = (1ULL << 63) + (f >> -ex);
    e = 0;
  } else {
    const uint64_t one = 1ULL << (63 - ex);
    m = f + one;
    e = ex;
    if (m < f) { /* 1 + y reached 2^(ex + 1) */
      m = (m >> 1) | 1ULL << 63;
      e = ex + 1;
    }
  }
  const int j = (int)(m >> 56) & 127;
  const uint64_t c = T->log_c[j];
  /* m c, 62 fraction bits below the product's top; r = m c - 1 with 64 */
  const uint64_t hi = __umul64hi(m, c), lo = m * c;
  /* m 2^-63 c 2^-63 = (hi:lo) 2^-126; minus 1 = 2^62 in hi */
  const int64_t rh = (int64_t)(hi - (1ULL << 62));
  const int64_t r = (int64_t)((uint64_t)rh << 2 | lo >> 62); /* 64 fraction bits, |r| < 2^-7 */
  const int64_t r2 = __mul64hi(r, r);
  const int64_t r3 = __mul64hi(r2, r), r4 = __mul64hi(r2, r2);
  const int64_t r5 = __mul64hi(r4, r);
  /* -r^2/2 + r^3/3 - r^4/4 + r^5/5 - r^6/6 + r^7/7 */
  int64_t s = r - (r2 >> 1) + __mul64hi(r3, 0x5555555555555555LL) - (r4 >> 2) + __mul64hi(r5, 0x3333333333333333LL);
  s -= __mul64hi(__mul64hi(r3, r3), 0x2aaaaaaaaaaaaaaaLL);
  s += __mul64hi(__mul64hi(r4, r3), 0x2492492492492492LL);
  /* sum with 58 fraction bits beside e ln 2: up to 2^6 */
  const uint64_t whole = (uint64_t)e * (IX_LN2_64 >> 7); /* 57 fraction bits */
  const int64_t part = (int64_t)(T->log_v[j]) + (s >> 1); /* 63 fraction bits */
  if (e == 0) return part <= 0 ? 0.0 : ix_frac_double((uint64_t)part);
  const uint64_t sum = whole + (uint64_t)(part >> 6); /* 57 fraction bits, below 2^63 */
  const int lz = __clzll((long long)sum);
  return ix_double(sum << lz, 6 - lz);
}

/* ln m of m 2^-63 in [1, 2), with 63 fraction bits: r = m c_j - 1 as above. */
__device__ __forceinline__ int64_t ix_log_mant(const IxTables* T, uint64_t m) {
  const int j = (int)(m >> 56) & 127;
  const uint64_t c = T->log_c[j];
  const uint64_t hi = __umul64hi(m, c), lo = m * c;
  const int64_t r = (int64_t)((hi - (1ULL << 62)) << 2 | lo >> 62); /* 64 fraction bits, |r| < 2^-7 */
  const int64_t r2 = __mul64hi(r, r);
  const int64_t r3 = __mul64hi(r2, r), r4 = __mul64hi(r2, r2);
  const int64_t r5 = __mul64hi(r4, r);
  int64_t s = r - (r2 >> 1) + __mul64hi(r3, 0x5555555555555555LL) - (r4 >> 2) + __mul64hi(r5, 0x3333333333333333LL);
  s -= __mul64hi(__mul64hi(r3, r3), 0x2aaaaaaaaaaaaaaaLL);
  s += __mul64hi(__mul64hi(r4, r3), 0x2492492492492492LL);
  return (int64_t)T->log_v[j] + (s >> 1);
}

/* log2 x with 52 fraction bits of a positive normal x, rounded (within 2^-53). */
__device__ __forceinline__ int64_t ix_log2(const IxTables* T, double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int e = (int)(b >> 52) - 1023;
  const int64_t v = ix_log_mant(T, ((b & 0xfffffffffffffULL) | 1ULL << 52) << 11);
  const int64_t f = __mul64hi(v, 0x5c551d94ae0bf85eLL); /* times 1/(2 ln 2): log2 m with 61 fraction bits */
  return ((int64_t)e << 52) + ((f + (1LL << 8)) >> 9);
}

/* The tables, formed once (0.1 ms where long double is done in software). */
inline const IxTables* ix_tables() {
  static const IxTables tables = [] {
    IxTables T;
    for (int j = 0; j < IX_EXP_N; ++j) T.exp2_t[j] = (uint64_t)rintl(exp2l(j / 128.0L) * 9223372036854775808.0L);
    for (int j = 0; j < IX_LOG_N; ++j) {
      const long double c = rintl(1024.0L / (1.0L + (j + 0.5L) / 128.0L)) / 1024.0L;
      T.log_c[j] = (uint64_t)(c * 9223372036854775808.0L);
      T.log_v[j] = (uint64_t)(-logl(c) * 9223372036854775808.0L);
    }
    return T;
  }();
  return &tables;
}

#endif /* LPG_IXMATH_CUH */
