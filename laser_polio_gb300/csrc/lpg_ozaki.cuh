/*
 * lpg_ozaki.cuh — double-precision matrix products on the tensor cores by
 * exact slicing (Ozaki, Ogita, Oishi, Rump, "Error-free transformations of
 * matrix multiplication by using fast routines of matrix multiplication",
 * Numerical Algorithms 59, 2012).
 *
 * C = A B, A given row by row and B column by column along the depth k.
 * Each row of A and column of B is scaled by a power of two to |x| < 1 and
 * cut into eight signed digits, x = sum_i d_i 2^-(6 + 7i), d_i an integer in
 * [-64, 64], which leaves at most 2^-56.  Digits are held as bf16 values
 * d_i 2^-7i (exact), so that tcgen05.mma forms every product d_i e_j
 * 2^-7(i+j) exactly, and the products of one diagonal i + j are summed in
 * one FP32 accumulator in TMEM: at most eight pairs of at most 2^12 over a
 * depth of at most 512 stay within 2^24 units, so those sums are exact
 * whatever their order.  Diagonal 8 (2^-56 and below) is added to the last
 * accumulator, where rounding is 2^-24 of terms of that size; what lies
 * beyond is dropped.  The epilogue adds the eight sums as integers and
 * rounds to a double once, scaled back by the two powers of two.
 *
 * What bounds it: the tensor core's reads of shared memory.  A slice of A is
 * multiplied with up to four slices of B at once (N = 256; their rows follow
 * one another as their diagonals do in TMEM), which took the products of a
 * stage from 3.4 to 1.7 us; loads and products in warps of their own took
 * a stage from 2.9 us to those 1.7.  Measured: 1095 x 774 x 774 in 70 us,
 * 774 x 774 x 1095 in 61, 270 x 4000 x 4000 in 358, 4000 x 4000 x 270 in 307
 * (double-float on the FP32 pipe: 311, 355, 2015 and 1821).  An element's
 * error is relative to its row's and column's largest, not to itself, so
 * k_oz_refine forms the elements again that are small beside those.
 *
 * Non-finite elements make their whole row or column scale NaN, and so
 * every element of C they take part in, as in a product that adds NaN.
 */
#ifndef LPG_OZAKI_CUH
#define LPG_OZAKI_CUH

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#define OZ_SLICES 8
#define OZ_BM 128 /* rows of C a tile: the lanes of TMEM */
#define OZ_BN 64  /* columns of C a tile: eight accumulators fill TMEM's 512 columns */
#define OZ_BK 32  /* depth of a stage: 64 bytes of bf16, one 64-byte swizzle row */
#define OZ_CHUNK (512 / OZ_BK) /* stages summed in TMEM before a drain (exactness, above) */
#define OZ_STAGES 2
#define OZ_DRAIN_WARPS 16
#define OZ_THREADS (32 * OZ_DRAIN_WARPS + 64) /* and a load warp and a product warp */
#define OZ_A_BYTES (OZ_SLICES * OZ_BM * OZ_BK * 2)
#define OZ_B_BYTES (OZ_SLICES * OZ_BN * OZ_BK * 2)
#define OZ_STAGE_BYTES (OZ_A_BYTES + OZ_B_BYTES)
#define OZ_SMEM (OZ_STAGES * OZ_STAGE_BYTES + 1024)
#define OZ_WAIT_POLLS (1 << 24) /* a wait gives up after so many polls, about 2.2 s (0.13 us each, measured) */
#define OZ_NAN_EXP 0x7fffffff

/* --- slicing --------------------------------------------------------------- */
/* The scale 2^e of a row or column from the largest magnitude's bits:
 * |x| < 2^e; OZ_NAN_EXP when an element is not finite. */
__device__ __forceinline__ int oz_exp(uint64_t max_bits) {
  const int b = (int)(max_bits >> 52);
  if (b >= 0x7ff) return OZ_NAN_EXP;
  return b - 1022 < -900 ? -900 : b - 1022;
}

__device__ __forceinline__ uint64_t oz_abs_bits(double x) {
  return (uint64_t)__double_as_longlong(x) & 0x7fffffffffffffffULL;
}

/* x times fac[k], where factors are given (the factor 1 told by its bits: a
 * comparison of doubles is an FP64 operation). */
__device__ __forceinline__ double oz_scaled(double x, const double* fac, int k) {
  if (!fac) return x;
  const double f = __ldg(fac + k);
  return __double_as_longlong(f) == 0x3ff0000000000000LL ? x : x * f;
}

/* The eight digits of x 2^-e as bf16 bits of d_i 2^-7i. */
__device__ __forceinline__ void oz_digits(double x, int e, uint16_t out[OZ_SLICES]) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const int ex = (int)(b >> 52 & 0x7ff);
  int64_t v = 0; /* rint(x 2^(55 - e)) */
  if (ex != 0 && e != OZ_NAN_EXP) {
    const uint64_t m = (b & 0xfffffffffffffULL) | 1ULL << 52;
    const int sh = 1020 + e - ex; /* >= -2 */
    if (sh <= 0) v = (int64_t)(m << -sh);
    else if (sh < 56) v = (int64_t)((m + (1ULL << (sh - 1))) >> sh);
    if (b >> 63) v = -v;
  }
#pragma unroll
  for (int i = OZ_SLICES - 1; i > 0; --i) {
    const int d = (int)((v + 64) & 127) - 64;
    v = (v - d) >> 7;
    const float f = (float)d * __uint_as_float((uint32_t)(127 - 7 * i) << 23);
    out[i] = (uint16_t)(__float_as_uint(f) >> 16);
  }
  out[0] = (uint16_t)(__float_as_uint((float)(int)v) >> 16);
}

#define OZ_SQ_BITS 13       /* fraction bits of the sums of squares */

/* |x| 2^-e as FP32, truncated; 0 below 2^-126 and for subnormal x. */
__device__ __forceinline__ float oz_scaled_abs(double x, int e) {
  const uint32_t h = (uint32_t)(oz_abs_bits(x) >> 32), l = (uint32_t)__double2loint(x);
  const int ex = (int)(h >> 20) - 1023 - e + 127;
  if (ex <= 0 || h < 0x100000u) return 0.0f;
  if (ex >= 255) return __uint_as_float(0x7f7fffffu);
  return __uint_as_float((uint32_t)ex << 23 | (h & 0xfffffu) << 3 | l >> 29);
}

/* The square of x 2^-e with OZ_SQ_BITS fraction bits, rounded up. */
__device__ __forceinline__ uint32_t oz_square(double x, int e) {
  const float f = oz_scaled_abs(x, e);
  return e == OZ_NAN_EXP || f == 0.0f ? 0u : (uint32_t)(f * f * (float)(1 << OZ_SQ_BITS)) + 1u;
}

/* max |x| of every row / column of src [R][C] (bits; the caller clears max). */
__global__ void __launch_bounds__(256) k_oz_row_max(int R, int C, const double* __restrict__ src, unsigned long long* max) {
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= R) return;
  unsigned long long m = 0;
  for (int c = lane; c < C; c += 32) {
    const unsigned long long v = oz_abs_bits(src[(size_t)r * C + c]);
    m = v > m ? v : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
    m = v > m ? v : m;
  }
  if (lane == 0) max[r] = m;
}

/* Sixteen rows of 256 columns a CTA, their loads in flight together; fac: a
 * factor for each row, or null. */
#define OZ_MAX_ROWS 16
__global__ void __launch_bounds__(256)
    k_oz_col_max(int R, int C, const double* __restrict__ src, const double* __restrict__ fac, unsigned long long* max) {
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= C) return;
  unsigned long long m = 0;
  const int r0 = blockIdx.y * OZ_MAX_ROWS;
  double x[OZ_MAX_ROWS];
#pragma unroll
  for (int q = 0; q < OZ_MAX_ROWS; ++q) x[q] = r0 + q < R ? src[(size_t)(r0 + q) * C + c] : 0.0;
#pragma unroll
  for (int q = 0; q < OZ_MAX_ROWS; ++q) {
    const unsigned long long v = oz_abs_bits(r0 + q < R ? oz_scaled(x[q], fac, r0 + q) : 0.0);
    m = v > m ? v : m;
  }
  atomicMax(&max[c], m);
}

/* dst [8][R][Kp] from src [gridDim.x][K], scaled by rows; two depths a
 * thread.  The scaled rows' sums of squares are added to sq. */
__global__ void __launch_bounds__(256)
    k_oz_slice_rows(int R, int K, int Kp, const double* __restrict__ src, const unsigned long long* __restrict__ max,
                    uint32_t* __restrict__ dst, uint32_t* __restrict__ sq) {
  const int r = blockIdx.x, k = 2 * (blockIdx.y * 256 + threadIdx.x);
  const int e = oz_exp(max[r]);
  const double x = k < K ? src[(size_t)r * K + k] : 0.0, y = k + 1 < K ? src[(size_t)r * K + k + 1] : 0.0;
  const uint32_t sum = __reduce_add_sync(0xffffffffu, oz_square(x, e) + oz_square(y, e));
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&sq[r], sum);
  if (k >= Kp) return;
  uint16_t a[OZ_SLICES], b[OZ_SLICES];
  oz_digits(x, e, a);
  oz_digits(y, e, b);
#pragma unroll
  for (int s = 0; s < OZ_SLICES; ++s)
    dst[((size_t)s * R + r) * (Kp / 2) + k / 2] = (uint32_t)a[s] | (uint32_t)b[s] << 16;
}

/* The first 32 gridDim.y depths of dst [8][C][Kp] from src [K][C] (times fac[k], when given), scaled by columns: 32 x 32 tiles turned in
 * shared memory, then two depths a thread, so that sixteen threads write one
 * 64-byte run.  The scaled columns' sums of squares are added to sq.  Bound by
 * the integer digit extraction and the writes. */
__global__ void __launch_bounds__(256)
    k_oz_slice_cols(int K, int C, int Kp, const double* __restrict__ src, const double* __restrict__ fac,
                    const unsigned long long* __restrict__ max, uint32_t* __restrict__ dst, uint32_t* __restrict__ sq) {
  __shared__ double s[32][33];
  const int c0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = k0 + ty + 8 * q, c = c0 + tx;
    s[ty + 8 * q][tx] = k < K && c < C ? oz_scaled(src[(size_t)k * C + c], fac, k) : 0.0;
  }
  __syncthreads();
  const int kp = threadIdx.x & 15;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int cl = (threadIdx.x >> 4) + 16 * q, c = c0 + cl;
    if (c >= C) continue;
    const int e = oz_exp(max[c]);
    uint16_t a[OZ_SLICES], b[OZ_SLICES];
    oz_digits(s[2 * kp][cl], e, a);
    oz_digits(s[2 * kp + 1][cl], e, b);
    const uint32_t sum = __reduce_add_sync(0xffffu << (threadIdx.x & 16), oz_square(s[2 * kp][cl], e) +
                                                                              oz_square(s[2 * kp + 1][cl], e));
    if (kp == 0 && sum) atomicAdd(&sq[c], sum);
#pragma unroll
    for (int i = 0; i < OZ_SLICES; ++i)
      dst[((size_t)i * C + c) * (Kp / 2) + k0 / 2 + kp] = (uint32_t)a[i] | (uint32_t)b[i] << 16;
  }
}

/* --- the product ------------------------------------------------------------ */
__device__ __forceinline__ uint32_t oz_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
/* Counted in polls, not in time: those do not go on while the context is
 * switched out or held by a debugger. */
__device__ __forceinline__ bool oz_wait(uint64_t* bar, uint32_t parity, const volatile int* fail, int polls) {
  for (int it = 0; it < polls; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(oz_smem(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (fail && *fail) return false;
  }
  return false;
}

__device__ __forceinline__ void oz_load(uint32_t dst, const CUtensorMap* map, int k, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst),
      "l"(map), "r"(k), "r"(row), "r"(0), "r"(oz_smem(bar))
      : "memory");
}

/* K-major operand tile in 64-byte swizzled rows: groups of eight rows 512
 * bytes apart; the low word advances by address / 16. */
__device__ __forceinline__ uint64_t oz_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

/* D FP32, A and B bf16, both K-major, M = 128, N = 64 per slice of B */
#define OZ_IDESC(slices) (1u << 4 | 1u << 7 | 1u << 10 | ((slices) * OZ_BN / 8) << 17 | (OZ_BM / 16) << 24)

__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void oz_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(oz_smem(bar))
               : "memory");
}

__device__ __forceinline__ void oz_ld8(uint32_t addr, float v[8]) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

/* (hi 2^28 + lo) 2^(e - 61) as a double, rounded to nearest (|hi| < 2^46,
 * |lo| < 2^60), by integer operations: FP64 ones would cost as much as the
 * tile's products. */
__device__ __forceinline__ double oz_double(int64_t hi, int64_t lo, int e) {
  int64_t h = hi + (lo >> 28);
  uint64_t l = (uint64_t)lo & 0xfffffffULL; /* value = h 2^28 + l */
  const bool neg = h < 0;
  if (neg) {
    h = l ? -h - 1 : -h;
    l = l ? (1ULL << 28) - l : 0;
  }
  const uint64_t u = (uint64_t)h;
  if ((u | l) == 0) return 0.0;
  uint64_t m;
  int top; /* the value's leading bit is 2^(top - 61 + e) */
  if (u >> 35) {
    const int lz = __clzll((long long)u);
    m = lz >= 28 ? (u << lz) | (l << (lz - 28)) : (u << lz) | (l >> (28 - lz));
    top = 63 - lz + 28;
  } else {
    m = u << 28 | l;
    const int lz = __clzll((long long)m);
    m <<= lz;
    top = 63 - lz;
  }
  const uint64_t r = m + (1ULL << 10);
  const bool carry = r < m;
  int ex = top - 61 + e + 1023 + (carry ? 1 : 0);
  uint64_t mant = carry ? 0 : (r >> 11) & 0xfffffffffffffULL;
  if (ex <= 0) {
    ex = 0;
    mant = 0;
  } else if (ex >= 0x7ff) {
    ex = 0x7ff;
    mant = 0;
  }
  return __longlong_as_double((long long)((neg ? 1ULL << 63 : 0) | (uint64_t)ex << 52 | mant));
}

struct OzArgs {
  int M, N, k_stages;     /* depth in stages of OZ_BK */
  int split, per_split;   /* depth slices, stages a slice */
  int tiles_n, tiles;
  int add;                /* to what C holds */
  int polls, stall;       /* a wait's limit; the load after which no more are issued (a test's; negative: none) */
  const unsigned long long *max_a, *max_b;
  double* C; /* [split][M][N] */
  double* err;
};

/* One (tile, depth slice) unit after another per CTA, one CTA an SM (TMEM
 * and shared memory are one CTA's).  A load warp keeps two stages of TMA
 * loads ahead, a product warp issues each stage's digit products (the queue
 * of issued products is short, so a thread that did both would load late),
 * and sixteen warps drain the accumulators.  Every wait is bounded and gives
 * up once another has: then *err is set, the products and loads in flight are
 * waited for (bounded) and the CTA gives its TMEM back and leaves. */
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, OzArgs G) {
  extern __shared__ uint8_t oz_raw[];
  __shared__ uint64_t full[OZ_STAGES], empty[OZ_STAGES], done, drained, quiet;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_fail;
  const uint32_t base = (oz_smem(oz_raw) + 1023u) & ~1023u;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < OZ_STAGES; ++s) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(&full[s])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(&empty[s])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(&done)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(oz_smem(&quiet)) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(oz_smem(&drained)), "r"(OZ_DRAIN_WARPS) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = 0;
  }
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(oz_smem(&s_tmem))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  const int units = G.tiles * G.split;
  int loads = 0; /* issued, by the load warp's first lane */

  if (warp == OZ_DRAIN_WARPS) { /* loads */
    if (lane == 0) {
      bool ok = true;
      for (int unit = blockIdx.x; ok && unit < units; unit += gridDim.x) {
        const int z = unit / G.tiles, tile = unit % G.tiles;
        const int k0 = z * G.per_split, k1 = min(G.k_stages, k0 + G.per_split);
        for (int k = k0; k < k1; ++k, ++loads) {
          const int s = loads % OZ_STAGES;
          if (loads == G.stall) {
            ok = false;
            break;
          }
          if (loads >= OZ_STAGES && !oz_wait(&empty[s], (uint32_t)(loads / OZ_STAGES - 1) & 1u, &s_fail, G.polls)) {
            s_fail = 1;
            ok = false;
            break;
          }
          const uint32_t dst = base + s * OZ_STAGE_BYTES;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(oz_smem(&full[s])),
                       "r"(OZ_STAGE_BYTES)
                       : "memory");
          oz_load(dst, &ta, k * OZ_BK, (tile / G.tiles_n) * OZ_BM, &full[s]);
          oz_load(dst + OZ_A_BYTES, &tb, k * OZ_BK, (tile % G.tiles_n) * OZ_BN, &full[s]);
        }
      }
    }
  } else if (warp == OZ_DRAIN_WARPS + 1) { /* products */
    if (lane == 0) {
      int n = 0, drains = 0;
      bool ok = true;
      for (int unit = blockIdx.x; ok && unit < units; unit += gridDim.x) {
        const int z = unit / G.tiles;
        const int k0 = z * G.per_split, k1 = min(G.k_stages, k0 + G.per_split);
        for (int kc = k0; ok && kc < k1; kc += OZ_CHUNK, ++drains) {
          if (drains > 0 && !oz_wait(&drained, (uint32_t)(drains - 1) & 1u, &s_fail, G.polls)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int ke = min(k1, kc + OZ_CHUNK);
          for (int k = kc; k < ke; ++k, ++n) {
            const int s = n % OZ_STAGES;
            if (!oz_wait(&full[s], (uint32_t)(n / OZ_STAGES) & 1u, &s_fail, G.polls)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t da = oz_desc(base + s * OZ_STAGE_BYTES);
            const uint64_t db = oz_desc(base + s * OZ_STAGE_BYTES + OZ_A_BYTES);
#pragma unroll 1
            for (int h = 0; h < OZ_BK / 16; ++h) {
              const uint32_t first = (k == kc && h == 0) ? 0u : 1u;
#pragma unroll
              for (int i = 0; i < OZ_SLICES; ++i) {
                const uint64_t ai = da + (uint64_t)((i * OZ_BM * OZ_BK * 2 + h * 32) >> 4);
                /* digits j .. j+c-1 of B in one instruction: their rows follow
                 * one another in shared memory as their diagonals do in TMEM */
#pragma unroll
                for (int j = 0; j < OZ_SLICES - i; j += 4) {
                  const int c = OZ_SLICES - i - j < 4 ? OZ_SLICES - i - j : 4;
                  oz_mma(tmem + (i + j) * OZ_BN, ai, db + (uint64_t)((j * OZ_BN * OZ_BK * 2 + h * 32) >> 4),
                         OZ_IDESC(c), i == 0 ? first : 1u);
                }
                if (i > 0) /* diagonal 8 */
                  oz_mma(tmem + (OZ_SLICES - 1) * OZ_BN, ai,
                         db + (uint64_t)(((OZ_SLICES - i) * OZ_BN * OZ_BK * 2 + h * 32) >> 4), OZ_IDESC(1), 1u);
              }
            }
            oz_commit(&empty[s]);
          }
          if (ok) oz_commit(&done);
        }
      }
      if (!ok) s_fail = 1;
    }
  } else { /* drains */
    int drains = 0;
    bool ok = true;
    for (int unit = blockIdx.x; ok && unit < units; unit += gridDim.x) {
      const int z = unit / G.tiles, tile = unit % G.tiles;
      const int k0 = z * G.per_split, k1 = min(G.k_stages, k0 + G.per_split);
      const int row = (tile / G.tiles_n) * OZ_BM + (warp & 3) * 32 + lane;
      const int col0 = (tile % G.tiles_n) * OZ_BN + (warp >> 2) * 16;
      double* Cz = G.C + (size_t)z * G.M * G.N;
      for (int kc = k0; ok && kc < k1; kc += OZ_CHUNK, ++drains) {
        ok = oz_wait(&done, (uint32_t)drains & 1u, &s_fail, G.polls);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          s_fail = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int ea = row < G.M ? oz_exp(G.max_a[row]) : 0;
        const bool even = (G.N & 1) == 0; /* rows then start 16-byte aligned */
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          int64_t hi[8], lo[8];
#pragma unroll
          for (int d = 0; d < OZ_SLICES; ++d) {
            float v[8];
            oz_ld8(tmem + ((uint32_t)((warp & 3) * 32) << 16) + d * OZ_BN + (warp >> 2) * 16 + g * 8, v);
            const float up = __uint_as_float((uint32_t)(127 + 7 * d) << 23);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const int q = __float2int_rn(v[c] * up);
              if (d == 0) hi[c] = (int64_t)q * (1 << 21);
              else if (d < 4) hi[c] += (int64_t)q * (1 << (21 - 7 * d));
              else if (d == 4) lo[c] = (int64_t)q * (1 << 21);
              else lo[c] += (int64_t)q * (1 << (7 * (7 - d)));
            }
          }
          if (g == 1) { /* the accumulators are read: the next products may start */
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(oz_smem(&drained)) : "memory");
          }
          if (row >= G.M) continue;
          const int col = col0 + g * 8;
          double* out = Cz + (size_t)row * G.N + col;
#pragma unroll
          for (int c = 0; c < 8; c += 2) {
            double w[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int eb = col + c + q < G.N ? oz_exp(G.max_b[col + c + q]) : 0;
              w[q] = ea == OZ_NAN_EXP || eb == OZ_NAN_EXP ? __longlong_as_double(0x7ff8000000000000LL)
                                                          : oz_double(hi[c + q], lo[c + q], ea + eb);
              if ((kc != k0 || G.add) && col + c + q < G.N) w[q] += out[c + q];
            }
            if (col + c + 1 < G.N && even) {
              *reinterpret_cast<double2*>(out + c) = make_double2(w[0], w[1]);
            } else {
              if (col + c < G.N) out[c] = w[0];
              if (col + c + 1 < G.N) out[c + 1] = w[1];
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (s_fail) { /* in a good run the drains have waited for every product, and the products for every load */
    if (tid == 0) *G.err = 1.0;
    if (warp == OZ_DRAIN_WARPS && lane == 0)
      for (int q = loads > OZ_STAGES ? loads - OZ_STAGES : 0; q < loads; ++q)
        oz_wait(&full[q % OZ_STAGES], (uint32_t)(q / OZ_STAGES) & 1u, nullptr, OZ_WAIT_POLLS);
    if (warp == OZ_DRAIN_WARPS + 1 && lane == 0) { /* the thread that issued the products */
      oz_commit(&quiet);
      oz_wait(&quiet, 0, nullptr, OZ_WAIT_POLLS);
    }
    __syncthreads();
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

/* --- elements the digits cannot hold ------------------------------------------ */
/* A digit product's element is off by about 2^-57 of its row's scale times
 * its column's, and a sum over the depth by e = 2^-56.8 sqrt(sum a^2 + sum
 * b^2) of them (a, b scaled to 1: a rounding of half of 2^-55 each, uniform).
 * Where the element itself is small beside the two scales — a wave that has
 * not reached the other's node, a flow across the map, one large node above
 * a background — that is too much of it.  So an element is kept only where
 * its summed terms are at least 2^45 e, so that it is off by at most 2^-45 of
 * them (rms) as any element of a product of FP32 pairs is (rms 2^-45, 2^-42
 * at worst, 774 terms).  |C| bounds the sum of the terms' magnitudes from
 * below, and equals it where no signs differ. */
#define OZ_KEEP 0x1.26p-12f /* 2^(45 - 56.8) */

/* sqrt(sum a^2 + sum b^2) */
__device__ __forceinline__ float oz_norm(uint32_t sa, uint32_t sb) {
  return sqrtf(((float)sa + (float)sb) * (1.0f / (1 << OZ_SQ_BITS)));
}

/* Whether an element whose value is c cannot stay as the digits gave it. */
__device__ __forceinline__ bool oz_small(double c, int ea, int eb, uint32_t sa, uint32_t sb) {
  if (ea == OZ_NAN_EXP || eb == OZ_NAN_EXP || sa == 0 || sb == 0) return false; /* NaN, or exactly 0 */
  return oz_scaled_abs(c, ea + eb) < OZ_KEEP * oz_norm(sa, sb);
}

/* x 2^(30 - e) as an FP32 pair: 24 bits cut off, the 29 below them rounded
 * (30: room below for what is small beside the scale). */
__device__ __forceinline__ float2 oz_pair(double x, int e) {
  const uint64_t b = oz_abs_bits(x);
  const int ex = (int)(b >> 52) - 1023 + 30 - e + 127;
  if (e == OZ_NAN_EXP || ex <= 0 || b >> 52 == 0) return make_float2(0.f, 0.f);
  const uint32_t sign = (uint32_t)(__double2hiint(x)) & 0x80000000u;
  const float hi = __uint_as_float(sign | (uint32_t)ex << 23 | (uint32_t)(b >> 29 & 0x7fffffu));
  const float low = (float)(uint32_t)(b & 0x1fffffffu); /* units of 2^(ex - 127 - 52) */
  const float unit = ex > 52 ? __uint_as_float((uint32_t)(ex - 52) << 23) : 0.f;
  return make_float2(hi, __uint_as_float(__float_as_uint(__fmul_rn(low, unit)) | sign));
}

/* (sh, sl) += a * b for FP32 pairs a, b: the exact product of the high
 * parts (Dekker, by FMA) plus the cross terms, added by Knuth's TwoSum. */
__device__ __forceinline__ void oz_pair_fma(float& sh, float& sl, float2 a, float2 b) {
  const float ph = __fmul_rn(a.x, b.x);
  float pl = __fmaf_rn(a.x, b.x, -ph);
  pl = __fmaf_rn(a.x, b.y, pl);
  pl = __fmaf_rn(a.y, b.x, pl);
  const float s = __fadd_rn(sh, ph);
  const float bp = __fsub_rn(s, sh);
  const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(s, bp)), __fsub_rn(ph, bp));
  sl = __fadd_rn(sl, __fadd_rn(err, pl));
  sh = s;
}

struct OzRefine {
  int M, N, K, split;
  const double *A, *B; /* A [M][K], or [K][M]; B [K][N], its row k times fac[k] where given */
  const double* fac;
  const unsigned long long *max_a, *max_b;
  const uint32_t *sq_a, *sq_b;
  double* C; /* [split][M][N] */
  unsigned long long* count; /* entries of the list; cleared by the caller */
  uint64_t* list;            /* elements m N + n; OZ_R_LIST for each tile */
};

#define OZ_R_THREADS 128
#define OZ_R_BM 32
#define OZ_R_BN 32
#define OZ_R_BK 32
#define OZ_R_LIST 64 /* elements of a tile formed one by one */

/* Adds the depth slices into the first one, and finds the elements that
 * oz_small names, a 32 x 32 tile a CTA.  Up to OZ_R_LIST of them go to the
 * list (k_oz_fix); where there are more, they are formed here by a product of
 * FP32 pairs over the tile's rows that have some, and over the depths at
 * which those rows have terms (a row of few infected nodes has few).  Bound
 * by reading C where nothing is small; by FP32 issue where all is: 774 nodes,
 * 365 ticks, 3 strains, waves that hardly overlap: 547 us for the flows (a
 * 32 x 64 tile: 677).  With k_oz_fix 16 and 17 us for the two products of
 * that size where 0.1% of the mixing's elements are small, 49 and 47 us of
 * 4000 nodes and 90 ticks; 133 us for the mixing of a recorded run's
 * aggregates, 5% of whose elements are small.  The list's line: a tile of 774
 * terms in pairs takes an SM about 20 us, an element in FP64 0.4 us. */
template <bool TRANS_A>
__global__ void __launch_bounds__(OZ_R_THREADS) k_oz_refine(OzRefine R) {
  __shared__ int s_ea[OZ_R_BM], s_eb[OZ_R_BN], s_count, s_need;
  __shared__ unsigned long long s_at;
  __shared__ uint32_t s_sa[OZ_R_BM], s_sb[OZ_R_BN], s_rows, s_some;
  __shared__ uint16_t s_list[OZ_R_LIST];
  const int tid = threadIdx.x, m0 = blockIdx.y * OZ_R_BM, n0 = blockIdx.x * OZ_R_BN;
  if (tid < OZ_R_BN) {
    const bool in = n0 + tid < R.N;
    s_eb[tid] = in ? oz_exp(R.max_b[n0 + tid]) : 0;
    s_sb[tid] = in ? R.sq_b[n0 + tid] : 0;
  } else if (tid < OZ_R_BN + OZ_R_BM) {
    const int r = tid - OZ_R_BN;
    const bool in = m0 + r < R.M;
    s_ea[r] = in ? oz_exp(R.max_a[m0 + r]) : 0;
    s_sa[r] = in ? R.sq_a[m0 + r] : 0;
  }
  if (tid == 0) s_count = s_rows = 0;
  __syncthreads();
  if (tid < 32) {
    const uint32_t top = max(s_sa[tid], s_sb[tid]);
    const uint32_t most = __reduce_max_sync(0xffffffffu, top);
    /* the biased exponent that an element scaled by 2^(ea + eb) needs at most */
    if (tid == 0) s_need = (int)(__float_as_uint(OZ_KEEP * oz_norm(most, most)) >> 23) - 127 + 1023 + 1;
  }
  __syncthreads();
  auto where = [&](int r, int c) { return (size_t)(m0 + r) * R.N + n0 + c; };
  auto small = [&](int r, int c) {
    return m0 + r < R.M && n0 + c < R.N && oz_small(R.C[where(r, c)], s_ea[r], s_eb[c], s_sa[r], s_sb[c]);
  };
  /* a thread's column is one, so that an element is first compared by its
   * exponent with the most that any of the tile could need; only those below
   * are looked at closely */
  const int c = tid % OZ_R_BN, r0 = tid / OZ_R_BN;
  const int need = s_need + (s_eb[c] == OZ_NAN_EXP ? 0 : s_eb[c]);
  if (n0 + c < R.N) {
    constexpr int PER = OZ_R_BM * OZ_R_BN / OZ_R_THREADS, STEP = OZ_R_THREADS / OZ_R_BN;
    double v[PER]; /* a slice's loads in flight together */
#pragma unroll
    for (int i = 0; i < PER; ++i) v[i] = m0 + r0 + i * STEP < R.M ? R.C[where(r0 + i * STEP, c)] : 0.0;
#pragma unroll 1
    for (int z = 1; z < R.split; ++z) {
      const double* Cz = R.C + z * ((size_t)R.M * R.N);
      double w[PER];
#pragma unroll
      for (int i = 0; i < PER; ++i) w[i] = m0 + r0 + i * STEP < R.M ? Cz[where(r0 + i * STEP, c)] : 0.0;
#pragma unroll
      for (int i = 0; i < PER; ++i) v[i] += w[i];
    }
    if (R.split > 1)
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if (m0 + r0 + i * STEP < R.M) R.C[where(r0 + i * STEP, c)] = v[i];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int r = r0 + i * STEP;
      if ((__double2hiint(v[i]) >> 20 & 0x7ff) - s_ea[r] >= need || m0 + r >= R.M) continue;
      if (!oz_small(v[i], s_ea[r], s_eb[c], s_sa[r], s_sb[c])) continue;
      const int at = atomicAdd(&s_count, 1);
      atomicOr(&s_rows, 1u << r);
      if (at < OZ_R_LIST) s_list[at] = (uint16_t)(r * OZ_R_BN + c);
    }
  }
  __syncthreads();
  const int todo = s_count;
  if (todo == 0) return;
  if (todo <= OZ_R_LIST) {
    if (tid == 0) s_at = atomicAdd(R.count, (unsigned long long)todo);
    __syncthreads();
    if (tid < todo) R.list[s_at + tid] = where(s_list[tid] / OZ_R_BN, s_list[tid] % OZ_R_BN);
    return;
  }
  __shared__ float2 sA[OZ_R_BK][OZ_R_BM + 1]; /* [k][m] */
  __shared__ float2 sB[OZ_R_BK][OZ_R_BN];     /* [k][n] */
  const int tx = tid & 15, ty = tid >> 4;
  float sh[4][2], sl[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) sh[i][j] = sl[i][j] = 0.f;
  const uint32_t rows = s_rows; /* the others' elements stay */
#pragma unroll 1
  for (int k0 = 0; k0 < R.K; k0 += OZ_R_BK) {
    __syncthreads();
    if (tid == 0) s_some = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < (OZ_R_BK * OZ_R_BM) / OZ_R_THREADS; ++q) {
      const int e = tid + q * OZ_R_THREADS;
      const int hi = e >> 5, lo = e & 31;
      /* consecutive threads read consecutive m, or consecutive k */
      const int k = TRANS_A ? hi : lo, m = TRANS_A ? lo : hi;
      float2 v = make_float2(0.f, 0.f);
      if (k0 + k < R.K && (rows >> m & 1u))
        v = oz_pair(R.A[TRANS_A ? (size_t)(k0 + k) * R.M + m0 + m : (size_t)(m0 + m) * R.K + k0 + k], s_ea[m]);
      sA[k][m] = v;
      const uint32_t some = __ballot_sync(0xffffffffu, v.x != 0.0f);
      if (lo == 0 && some) atomicOr(&s_some, TRANS_A ? 1u << k : some);
    }
    __syncthreads();
    const uint32_t some = s_some; /* the depths at which some row has a term: few where few nodes are infected */
    if (some == 0) continue;
#pragma unroll
    for (int q = 0; q < (OZ_R_BK * OZ_R_BN) / OZ_R_THREADS; ++q) {
      const int e = tid + q * OZ_R_THREADS;
      const int k = e >> 5, n = e & 31;
      float2 v = make_float2(0.f, 0.f);
      if ((some >> k & 1u) && n0 + n < R.N)
        v = oz_pair(oz_scaled(R.B[(size_t)(k0 + k) * R.N + n0 + n], R.fac, k0 + k), s_eb[n]);
      sB[k][n] = v;
    }
    __syncthreads();
    auto add = [&](int q) {
      float2 av[4], bv[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sA[q][ty + 8 * i];
#pragma unroll
      for (int j = 0; j < 2; ++j) bv[j] = sB[q][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) oz_pair_fma(sh[i][j], sl[i][j], av[i], bv[j]);
    };
    if (some == 0xffffffffu) {
#pragma unroll 4
      for (int q = 0; q < OZ_R_BK; ++q) add(q);
    } else {
#pragma unroll 1
      for (uint32_t left = some; left; left &= left - 1) add(__ffs(left) - 1);
    }
    /* renormalise each pair (Fast2Sum: |sh| >= |sl|) so that sl stays small */
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float t = __fadd_rn(sh[i][j], sl[i][j]);
        sl[i][j] = __fsub_rn(sl[i][j], __fsub_rn(t, sh[i][j]));
        sh[i][j] = t;
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = ty + 8 * i, c = tx + 16 * j;
      if (small(r, c)) R.C[where(r, c)] = scalbn((double)sh[i][j] + (double)sl[i][j], s_ea[r] + s_eb[c] - 60);
    }
}

/* The listed elements in FP64, a CTA each; a warp each where there are more
 * than OZ_F_WARPS a CTA.  Where terms may cancel (TRANS_A: dL/du has both
 * signs) an element is given up as soon as the terms' magnitudes show that it
 * is good.  Bound by the latency of the column's reads, a sector each, and
 * with many elements by their number: then a warp reads B only where A is not
 * 0 (few nodes infected is what makes many elements small). */
#define OZ_F_WARPS 2
template <bool TRANS_A, int THREADS>
__device__ __forceinline__ void oz_fix_one(const OzRefine& R, size_t at, double* s_acc, float* s_mag) {
  constexpr bool CTA = THREADS > 32;
  const int t = threadIdx.x % THREADS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t m = at / R.N, n = at % R.N;
  const int ea = oz_exp(R.max_a[m]), eb = oz_exp(R.max_b[n]);
  const float keep = OZ_KEEP * oz_norm(R.sq_a[m], R.sq_b[n]);
  const double *a = R.A + (TRANS_A ? m : m * R.K), *b = R.B + n;
  double acc = 0.0;
  float mag = 0.f, all = 0.f;
  for (int k0 = 0; k0 < R.K && !(all >= keep); k0 += 8 * THREADS) { /* all: the same in every thread */
    double x[8], y[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * THREADS + t;
      x[u] = k < R.K ? a[TRANS_A ? (size_t)k * R.M : (size_t)k] : 0.0;
    }
    unsigned some = 0xffu; /* bit u: a term of some lane */
    if (!CTA) {
      some = 0;
#pragma unroll
      for (int u = 0; u < 8; ++u) some |= (unsigned)__any_sync(0xffffffffu, oz_abs_bits(x[u]) != 0) << u;
    }
    if (some == 0) continue;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * THREADS + t;
      y[u] = (some >> u & 1u) && k < R.K ? b[(size_t)k * R.N] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u * THREADS + t;
      if (!(some >> u & 1u)) continue;
      if (k < R.K) y[u] = oz_scaled(y[u], R.fac, k);
      acc = __fma_rn(x[u], y[u], acc);
      if (TRANS_A) mag += oz_scaled_abs(x[u], ea) * oz_scaled_abs(y[u], eb);
    }
    if (TRANS_A) {
      all = mag;
      for (int o = 16; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
      if (CTA) {
        if (lane == 0) s_mag[warp] = all;
        __syncthreads();
        all = (s_mag[0] + s_mag[1]) + (s_mag[2] + s_mag[3]);
        __syncthreads();
      }
    }
  }
  if (all >= keep) return;
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (CTA) {
    __syncthreads();
    if (lane == 0) s_acc[warp] = acc;
    __syncthreads();
    acc = (s_acc[0] + s_acc[1]) + (s_acc[2] + s_acc[3]);
  }
  if (t == 0) R.C[at] = acc;
}

template <bool TRANS_A>
__global__ void __launch_bounds__(OZ_R_THREADS) k_oz_fix(OzRefine R) {
  __shared__ double s_acc[OZ_R_THREADS / 32];
  __shared__ float s_mag[OZ_R_THREADS / 32];
  constexpr int WARPS = OZ_R_THREADS / 32;
  const unsigned long long todo = *R.count;
  if (todo <= (unsigned long long)OZ_F_WARPS * gridDim.x) {
    for (unsigned long long q = blockIdx.x; q < todo; q += gridDim.x)
      oz_fix_one<TRANS_A, OZ_R_THREADS>(R, R.list[q], s_acc, s_mag);
  } else {
    for (unsigned long long q = (unsigned long long)blockIdx.x * WARPS + (threadIdx.x >> 5); q < todo;
         q += (unsigned long long)gridDim.x * WARPS)
      oz_fix_one<TRANS_A, 32>(R, R.list[q], s_acc, s_mag);
  }
}

/* --- host side -------------------------------------------------------------- */
inline dim3 oz_col_grid(int R, int C) { return dim3((C + 255) / 256, (R + OZ_MAX_ROWS - 1) / OZ_MAX_ROWS); }

/* The tensor map of slices [8][rows][Kp] with boxes of box_rows rows; false
 * when the driver entry point is missing or refuses. */
inline bool oz_map(CUtensorMap* map, void* slices, int rows, int Kp, int box_rows) {
  typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return false;
  const cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, OZ_SLICES};
  const cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)rows * Kp * 2};
  const cuuint32_t box[3] = {OZ_BK, (cuuint32_t)box_rows, OZ_SLICES}, es[3] = {1, 1, 1};
  return ((Encode)fn)(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, slices, dims, strides, box, es,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

/* Depth slices: the count up to max_split that minimises the waves of units
 * times the stages (and a drain, about three stages' time) of each. */
inline void oz_plan(OzArgs* G, int nsm, int max_split) {
  G->tiles_n = (G->N + OZ_BN - 1) / OZ_BN;
  G->tiles = ((G->M + OZ_BM - 1) / OZ_BM) * G->tiles_n;
  long best = -1;
  for (int s = 1; s <= max_split && s <= G->k_stages; ++s) {
    const int per = (G->k_stages + s - 1) / s, n = (G->k_stages + per - 1) / per;
    const long waves = ((long)G->tiles * n + nsm - 1) / nsm;
    const long cost = waves * (per + 3 * ((per + OZ_CHUNK - 1) / OZ_CHUNK));
    if (best < 0 || cost < best) {
      best = cost;
      G->split = n;
      G->per_split = per;
    }
  }
}

inline cudaError_t oz_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const OzArgs& G, int nsm, cudaStream_t st) {
  if (G.polls <= 0) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM);
  if (e != cudaSuccess) return e;
  const int units = G.tiles * G.split;
  k_oz_gemm<<<units < nsm ? units : nsm, OZ_THREADS, OZ_SMEM, st>>>(ta, tb, G);
  return cudaGetLastError();
}

/* Entries of an M x N product's list. */
inline size_t oz_list(int M, int N) {
  return (size_t)OZ_R_LIST * ((N + OZ_R_BN - 1) / OZ_R_BN) * ((M + OZ_R_BM - 1) / OZ_R_BM);
}

template <bool TRANS_A>
inline cudaError_t oz_refine(const OzRefine& R, int nsm, cudaStream_t st) {
  k_oz_refine<TRANS_A><<<dim3((R.N + OZ_R_BN - 1) / OZ_R_BN, (R.M + OZ_R_BM - 1) / OZ_R_BM), OZ_R_THREADS, 0, st>>>(R);
  k_oz_fix<TRANS_A><<<8 * nsm, OZ_R_THREADS, 0, st>>>(R);
  return cudaGetLastError();
}

#endif /* LPG_OZAKI_CUH */
