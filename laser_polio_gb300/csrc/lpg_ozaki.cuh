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
 * (double-float on the FP32 pipe: 311, 355, 2015 and 1821); error 1e-16 of
 * the summed terms, rms.  An element's error is relative to its row's and
 * column's largest, not to itself.
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
#define OZ_WAIT_NS 1000000000ULL /* a wait gives up after a second */
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

/* dst [8][R][Kp] from src [R][K], scaled by rows; two depths a thread. */
__global__ void __launch_bounds__(256)
    k_oz_slice_rows(int R, int K, int Kp, const double* __restrict__ src, const unsigned long long* __restrict__ max,
                    uint32_t* __restrict__ dst) {
  const int r = blockIdx.x, k = 2 * (blockIdx.y * 256 + threadIdx.x);
  if (k >= Kp) return;
  const int e = oz_exp(max[r]);
  uint16_t a[OZ_SLICES], b[OZ_SLICES];
  oz_digits(k < K ? src[(size_t)r * K + k] : 0.0, e, a);
  oz_digits(k + 1 < K ? src[(size_t)r * K + k + 1] : 0.0, e, b);
#pragma unroll
  for (int s = 0; s < OZ_SLICES; ++s)
    dst[((size_t)s * R + r) * (Kp / 2) + k / 2] = (uint32_t)a[s] | (uint32_t)b[s] << 16;
}

/* dst [8][C][Kp] from src [K][C] (times fac[k], when given), scaled by columns: 32 x 32 tiles turned in
 * shared memory, then two depths a thread, so that sixteen threads write one
 * 64-byte run.  Bound by the integer digit extraction and the writes. */
__global__ void __launch_bounds__(256)
    k_oz_slice_cols(int K, int C, int Kp, const double* __restrict__ src, const double* __restrict__ fac,
                    const unsigned long long* __restrict__ max, uint32_t* __restrict__ dst) {
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
#pragma unroll
    for (int i = 0; i < OZ_SLICES; ++i)
      dst[((size_t)i * C + c) * (Kp / 2) + k0 / 2 + kp] = (uint32_t)a[i] | (uint32_t)b[i] << 16;
  }
}

/* --- the product ------------------------------------------------------------ */
__device__ __forceinline__ uint32_t oz_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool oz_wait(uint64_t* bar, uint32_t parity, const volatile int* fail) {
  uint64_t t0 = 0;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(oz_smem(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    if (t0 == 0) t0 = t;
    else if (t - t0 > OZ_WAIT_NS || *fail) return false;
  }
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
  const unsigned long long *max_a, *max_b;
  double* C; /* [split][M][N] */
  double* err;
};

/* One (tile, depth slice) unit after another per CTA, one CTA an SM (TMEM
 * and shared memory are one CTA's).  A load warp keeps two stages of TMA
 * loads ahead, a product warp issues each stage's digit products (the queue
 * of issued products is short, so a thread that did both would load late),
 * and sixteen warps drain the accumulators.  Every wait is bounded and gives
 * up once another has: then *err is set, the loads in flight are waited for
 * (bounded) and the CTA gives its TMEM back and leaves. */
__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, OzArgs G) {
  extern __shared__ uint8_t oz_raw[];
  __shared__ uint64_t full[OZ_STAGES], empty[OZ_STAGES], done, drained;
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

  if (warp == OZ_DRAIN_WARPS) { /* loads */
    if (lane == 0) {
      int n = 0;
      bool ok = true;
      for (int unit = blockIdx.x; ok && unit < units; unit += gridDim.x) {
        const int z = unit / G.tiles, tile = unit % G.tiles;
        const int k0 = z * G.per_split, k1 = min(G.k_stages, k0 + G.per_split);
        for (int k = k0; k < k1; ++k, ++n) {
          const int s = n % OZ_STAGES;
          if (n >= OZ_STAGES && !oz_wait(&empty[s], (uint32_t)(n / OZ_STAGES - 1) & 1u, &s_fail)) {
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
      /* nothing may land after the CTA has left (in a good run the products have waited for every load) */
      if (!ok) {
        const int never = 0;
        for (int q = n > OZ_STAGES ? n - OZ_STAGES : 0; q < n; ++q)
          oz_wait(&full[q % OZ_STAGES], (uint32_t)(q / OZ_STAGES) & 1u, &never);
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
          if (drains > 0 && !oz_wait(&drained, (uint32_t)(drains - 1) & 1u, &s_fail)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int ke = min(k1, kc + OZ_CHUNK);
          for (int k = kc; k < ke; ++k, ++n) {
            const int s = n % OZ_STAGES;
            if (!oz_wait(&full[s], (uint32_t)(n / OZ_STAGES) & 1u, &s_fail)) {
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
        ok = oz_wait(&done, (uint32_t)drains & 1u, &s_fail);
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
              if (kc != k0 && col + c + q < G.N) w[q] += out[c + q];
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
  if (tid == 0 && s_fail) *G.err = 1.0;
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
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
  cudaError_t e = cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM);
  if (e != cudaSuccess) return e;
  const int units = G.tiles * G.split;
  k_oz_gemm<<<units < nsm ? units : nsm, OZ_THREADS, OZ_SMEM, st>>>(ta, tb, G);
  return cudaGetLastError();
}

#endif /* LPG_OZAKI_CUH */
