/*
 * lpg_init_fast.cuh — the initialisation's timers and heterogeneity on the
 * FP32 pipe, with the same bits as the FP64 definitions of lpg_init.h.
 *
 * The definitions are double precision, and the GB300 issues about two FP64
 * operations per clock per SM against 128 FP32 ones: at 2.3e8 slots they
 * took 440 ms (timers) and 247 ms (heterogeneity), all of it FP64 issue.
 * What they store is small: whole days (int8) and FP32 values.  So each
 * value is formed here in FP32 (timers) or as an FP32 pair hi + lo
 * (heterogeneity) together with a bound on its distance from the FP64
 * result, and stored only when every decision on the way (a rejection, the
 * day it falls on, the FP32 value it rounds to) comes out the same anywhere
 * within that bound.  A slot where one does not (0.1-0.5% of them) is left
 * with a mark no finished slot carries (infection timer -1, risk -1), and
 * k_init_fix fills the marked slots with lpg_init.h's own functions.
 *
 * Work layout.  A CTA takes 1024 slots.  The first Philox block settles
 * most draws (a polar normal accepts 78.5% of its tries; the block holds
 * two); the others are queued in shared memory and finished by full warps,
 * so that a warp does not run every lane through the longest lane's blocks.
 */
#ifndef LPG_INIT_FAST_CUH
#define LPG_INIT_FAST_CUH

#include "lpg_init.h"

#define FI_TILE 1024
#define FI_THREADS 256
#define FI_FIX_TILE 16384

enum { FI_REJECT = 0, FI_OK = 1, FI_UNSURE = 2 };

/* One timer distribution: kinds with an FP32 form (fi_dist_of). */
struct FiDist {
  int32_t kind;
  float d, c, scale; /* gamma: Marsaglia-Tsang's d and c, d * scale */
  float mu, sg;      /* lognormal: of the normal underneath */
  float value;       /* constant */
  int32_t n_thr;     /* Poisson: thresholds on the 53-bit uniform */
  const uint64_t* thr;
};

__device__ __forceinline__ uint32_t fi_hi32(uint64_t w) { return (uint32_t)(w >> 32); }
/* 2u - 1 and u of a draw from its top 32 bits (the 21 bits below them add
 * at most 2^-31), rounded to FP32. */
__device__ __forceinline__ float fi_signed(uint32_t h) { return (float)(int32_t)(h ^ 0x80000000u) * 0x1.0p-31f; }
__device__ __forceinline__ float fi_unit(uint32_t h) { return (float)h * 0x1.0p-32f; }

/* One try of the polar method in FP32: the normal x and a bound on its
 * error.  q = u^2 + v^2 carries 2^-23 relative, so x = u sqrt(-2 ln q / q)
 * is off by at most about 2^-23.5 / sqrt(-ln q) + 2^-22 |x|: below 2^-18.5
 * for -ln q >= 2^-8 and 2^-16.5 down to 2^-14, doubled here.  Outside
 * [2^-14, 1 - 2^-14] the decision is left to FP64. */
__device__ __forceinline__ int fi_polar(uint32_t hu, uint32_t hv, float* x, float* err) {
  const float u = fi_signed(hu), v = fi_signed(hv);
  const float q = __fmaf_rn(u, u, __fmul_rn(v, v));
  if (q >= 1.0f + 0x1.0p-18f) return FI_REJECT;
  if (q > 1.0f - 0x1.0p-14f || q < 0x1.0p-14f) return FI_UNSURE;
  *x = u * sqrtf(-2.0f * logf(q) / q);
  *err = q > 1.0f - 0x1.0p-8f ? 0x1.0p-15f : 0x1.0p-17f;
  return FI_OK;
}

/* floor(v) when every value within err of v has the same floor. */
__device__ __forceinline__ int fi_floor(float v, float err, int* n) {
  const float f = floorf(v), r = v - f;
  *n = (int)f;
  return v < 0x1.0p20f && r > err && 1.0f - r > err ? FI_OK : FI_UNSURE;
}

__device__ __forceinline__ int fi_lognormal(const FiDist& D, float x, float ex, int* n) {
  const float a = __fmaf_rn(D.sg, x, D.mu);
  const float v = expf(a);
  return fi_floor(v, v * (D.sg * ex + (fabsf(a) + fabsf(D.mu) + 4.0f) * 0x1.0p-22f), n);
}

/* Marsaglia-Tsang's test of the normal x with the uniform of top bits hu.
 * The squeeze accepts a subset of what the logarithmic test accepts, so a
 * draw near the squeeze's edge may go to the logarithmic test. */
__device__ __forceinline__ int fi_gamma(const FiDist& D, float x, float ex, uint32_t hu, int* n) {
  const float v1 = __fmaf_rn(D.c, x, 1.0f);
  if (v1 < 0.05f) return FI_UNSURE; /* v1 <= 0 would leave the uniform unused */
  const float v = v1 * v1 * v1;
  const float u = fi_unit(hu), x2 = x * x;
  const float ev = 3.0f * v1 * v1 * D.c * ex + v * 0x1.0p-21f;
  if (!(u < 1.0f - 0.0331f * (x2 * x2) - 0x1.0p-12f)) {
    if (u < 0x1.0p-12f) return FI_UNSURE;
    const float lu = logf(u), lv = logf(v);
    const float rhs = __fmaf_rn(D.d, (1.0f - v) + lv, 0.5f * x2);
    const float e = D.d * (fabsf(1.0f / v - 1.0f) * ev + (1.0f + v + fabsf(lv)) * 0x1.0p-21f) + fabsf(x) * ex +
                    (x2 + fabsf(lu) + 1.0f) * 0x1.0p-20f;
    if (lu > rhs + e) return FI_REJECT;
    if (!(lu < rhs - e)) return FI_UNSURE;
  }
  const float g = D.scale * v;
  return fi_floor(g, D.scale * ev + g * 0x1.0p-21f, n);
}

/* The next place of a shared list, one atomic per warp. */
__device__ __forceinline__ int fi_place(int* count) {
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
  int base = 0;
  if (lane == lead) base = atomicAdd(count, __popc(m));
  return __shfl_sync(m, base, lead) + __popc(m & ((1u << lane) - 1u));
}

/* A draw still open after its first block: 0 nothing yet, 1 a normal waits
 * for its uniform (carry = the normal, err its bound's class), 2 one word
 * of the first block is unused (carry = its top bits). */
struct FiOpen {
  uint32_t id; /* stream << 16 | state << 20 | err class << 22 | slot in the tile */
  uint32_t carry;
};

__device__ __forceinline__ int fi_pt(int days, int e, int i) {
  int n = days - e;
  n = n < 0 ? 0 : n;
  return n > i ? i : n;
}
/* lpg_trunc_i8 of a non-negative whole number, then the clip at 0. */
__device__ __forceinline__ int fi_i8(int n) {
  const int b = (int)(int8_t)(uint8_t)(uint32_t)n;
  return b < 0 ? 0 : b;
}

/* Days of stream b in 15 bits: the exposure and infection timers keep the
 * low byte, the time to paralysis is clipped at 127 days or below. */
__device__ __forceinline__ int fi_days(int n, int b) { return b == 2 ? min(n, 0x7fff) : n & 0x7fff; }

struct FiTimers {
  uint64_t seed;
  int64_t capacity;
  FiDist d[3];
  int8_t *et, *it, *pt;
};

/* Bound by integer (Philox) issue: 3 blocks a slot, and about 2 more for the
 * open draws.  2.31e8 slots, gamma, gamma, lognormal: 19.6 ms with
 * k_init_fix; the FP64 pass took 442 ms. */
__global__ void __launch_bounds__(FI_THREADS) k_init_timers_fast(FiTimers A) {
  __shared__ FiOpen s_open[3 * FI_TILE];
  __shared__ int16_t s_n[3][FI_TILE]; /* whole days (fi_days), or -1 for unsure */
  __shared__ int s_count;
  const int64_t tiles = (A.capacity + FI_TILE - 1) / FI_TILE;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t i0 = tile * FI_TILE;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (int b = 0; b < 3; ++b) {
      const FiDist& D = A.d[b];
      for (int o = threadIdx.x; o < FI_TILE; o += FI_THREADS) {
        const int64_t i = i0 + o;
        if (i >= A.capacity) break;
        int n = 0, st = FI_UNSURE;
        FiOpen open;
        open.id = (uint32_t)b << 16 | (uint32_t)o;
        open.carry = 0;
        bool pending = false;
        if (D.kind == LPG_DIST_CONSTANT) {
          n = (int)D.value;
          st = FI_OK;
        } else {
          uint64_t c[4] = {(uint64_t)i, (uint64_t)b, (uint64_t)LPG_P_INIT_TIMER << 32, 0};
          lpg_philox4x64_10(c, A.seed, LPG_KEY_TAG);
          if (D.kind == LPG_DIST_POISSON) {
            const uint64_t m = c[0] >> 11;
            int k = 0;
            while (k < D.n_thr && m > __ldg(&D.thr[k])) ++k;
            n = k;
            st = k < D.n_thr ? FI_OK : FI_UNSURE;
          } else {
            float x = 0.f, ex = 0.f;
            st = fi_polar(fi_hi32(c[0]), fi_hi32(c[1]), &x, &ex);
            if (st == FI_OK) {
              if (D.kind == LPG_DIST_LOGNORMAL) {
                st = fi_lognormal(D, x, ex, &n);
              } else {
                st = fi_gamma(D, x, ex, fi_hi32(c[2]), &n);
                if (st == FI_REJECT) {
                  pending = true;
                  open.id |= 2u << 20;
                  open.carry = fi_hi32(c[3]);
                }
              }
            } else if (st == FI_REJECT) {
              st = fi_polar(fi_hi32(c[2]), fi_hi32(c[3]), &x, &ex);
              if (st == FI_OK && D.kind == LPG_DIST_LOGNORMAL) {
                st = fi_lognormal(D, x, ex, &n);
              } else if (st != FI_UNSURE) {
                pending = true;
                if (st == FI_OK) {
                  open.id |= 1u << 20 | (ex > 0x1.0p-16f ? 1u << 22 : 0u);
                  open.carry = __float_as_uint(x);
                }
              }
            }
          }
        }
        s_n[b][o] = (int16_t)(st == FI_OK ? fi_days(n, b) : -1);
        if (pending) s_open[fi_place(&s_count)] = open;
      }
    }
    __syncthreads();
    const int todo = s_count;
    for (int q = threadIdx.x; q < todo; q += FI_THREADS) {
      const FiOpen open = s_open[q];
      const int o = (int)(open.id & 0xffffu), b = (int)(open.id >> 16 & 3u), state = (int)(open.id >> 20 & 3u);
      const FiDist& D = A.d[b];
      const bool gamma = D.kind == LPG_DIST_GAMMA;
      float x = 0.f, ex = 0.f;
      bool have_x = state == 1, have_u = state == 2;
      uint32_t hu = open.carry;
      if (have_x) {
        x = __uint_as_float(open.carry);
        ex = open.id >> 22 & 1u ? 0x1.0p-15f : 0x1.0p-17f;
      }
      int n = 0, st = FI_REJECT;
      for (int blk = 1; blk < 32 && st == FI_REJECT; ++blk) {
        uint64_t c[4] = {(uint64_t)(i0 + o), (uint64_t)b, (uint64_t)LPG_P_INIT_TIMER << 32, (uint64_t)blk};
        lpg_philox4x64_10(c, A.seed, LPG_KEY_TAG);
        uint32_t h[4] = {fi_hi32(c[0]), fi_hi32(c[1]), fi_hi32(c[2]), fi_hi32(c[3])};
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          if (st != FI_REJECT) break;
          if (have_x) { /* the word is the gamma test's uniform */
            st = fi_gamma(D, x, ex, h[w], &n);
            have_x = false;
          } else if (!have_u) {
            hu = h[w];
            have_u = true;
          } else {
            have_u = false;
            const int p = fi_polar(hu, h[w], &x, &ex);
            if (p == FI_UNSURE) st = FI_UNSURE;
            if (p == FI_OK) {
              if (gamma) have_x = true;
              else st = fi_lognormal(D, x, ex, &n);
            }
          }
        }
      }
      s_n[b][o] = (int16_t)(st == FI_OK ? fi_days(n, b) : -1);
    }
    __syncthreads();
    for (int o = threadIdx.x; o < FI_TILE; o += FI_THREADS) {
      const int64_t i = i0 + o;
      if (i >= A.capacity) break;
      const int ne = s_n[0][o], ni = s_n[1][o], np = s_n[2][o];
      if (ne < 0 || ni < 0 || np < 0) {
        A.it[i] = -1; /* for k_init_fix */
        continue;
      }
      const int e = fi_i8(ne), t = fi_i8(ni);
      A.et[i] = (int8_t)e;
      A.it[i] = (int8_t)t;
      A.pt[i] = (int8_t)fi_pt(np, e, t);
    }
    __syncthreads();
  }
}

/* --- FP32 pairs ------------------------------------------------------------ */
__device__ __forceinline__ float2 ff_fast2(float a, float b) { /* |a| >= |b| or a = 0 */
  const float s = __fadd_rn(a, b);
  return make_float2(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ float2 ff_two(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return make_float2(s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb)));
}
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
  const float2 s = ff_two(a.x, b.x);
  return ff_fast2(s.x, __fadd_rn(s.y, __fadd_rn(a.y, b.y)));
}
__device__ __forceinline__ float2 ff_mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = __fmaf_rn(a.x, b.x, -p);
  e = __fmaf_rn(a.x, b.y, e);
  e = __fmaf_rn(a.y, b.x, e);
  return ff_fast2(p, e);
}
__device__ __forceinline__ float2 ff_div(float2 a, float2 b) {
  const float r = __frcp_rn(b.x), q = __fmul_rn(a.x, r);
  float rem = __fmaf_rn(-q, b.x, a.x);
  rem = __fadd_rn(rem, __fmaf_rn(-q, b.y, a.y));
  return ff_fast2(q, __fmul_rn(rem, r));
}
__device__ __forceinline__ float2 ff_sqrt(float2 a) {
  const float y = rsqrtf(a.x), s = __fmul_rn(a.x, y);
  const float rem = __fadd_rn(__fmaf_rn(-s, s, a.x), a.y);
  return ff_fast2(s, __fmul_rn(__fmul_rn(rem, 0.5f), y));
}

/* Tables of the pair functions, formed on the host (fi_tables): ln c_j for
 * the reciprocals c_j of 129 points of [0.75, 1.5), 2^(j/64), and the series
 * of -ln(1 - Phi) about 32 points a unit of [-3.5, 5.5]. */
#define FI_LOG_N 129
#define FI_EXP_N 64
#define FI_G_LO (-3.5f)
#define FI_G_HI 5.5f
#define FI_G_STEPS 32
#define FI_G_N 290
struct FiTables {
  float4 log_c[FI_LOG_N];  /* c, -ln c (hi, lo), unused */
  float2 exp_t[FI_EXP_N];
  float4 g[FI_G_N][3]; /* (c0, c1), (c2, c3 c4), (c5 c6, unused) */
};

/* ln q for 2^-12 <= q <= 1 - 2^-12: q = 2^e m, r = m c_j - 1 with the
 * product's low part kept, |r| <= 2^-8; the series beyond r in FP32
 * (below 2^-40 absolute). */
__device__ __forceinline__ float2 ff_log(const FiTables* T, float2 q) {
  const uint32_t b = __float_as_uint(q.x);
  int e = (int)(b >> 23) - 127;
  const uint32_t mant = b & 0x7fffffu;
  const int j = (int)((mant + 0x8000u) >> 16); /* m near 1 + j/128 */
  if (j >= 64) e += 1;                         /* then m is in [0.75, 1] */
  const float s = __uint_as_float((uint32_t)(127 - e) << 23);
  const float mh = q.x * s, ml = q.y * s;
  const float4 c = T->log_c[j];
  const float p = __fmul_rn(mh, c.x);
  const float pl = __fmaf_rn(ml, c.x, __fmaf_rn(mh, c.x, -p));
  const float2 r = ff_fast2(__fsub_rn(p, 1.0f), pl);
  const float t = r.x;
  float poly = __fmaf_rn(t, 0.2f, -0.25f);
  poly = __fmaf_rn(t, poly, 0x1.555556p-2f);
  poly = __fmaf_rn(t, poly, -0.5f);
  poly = __fmul_rn(__fmul_rn(t, t), poly);
  const float fe = (float)e;
  /* ln 2 in 15, 24 and 24 bits: e times the first part is exact */
  const float e2 = __fmul_rn(fe, 0x1.7f7d1cp-20f);
  float2 l = ff_two(__fmul_rn(fe, 0x1.62e4p-1f), e2);
  l.y = __fadd_rn(l.y, __fmaf_rn(fe, 0x1.ef357ap-45f, __fmaf_rn(fe, 0x1.7f7d1cp-20f, -e2)));
  l = ff_add(l, make_float2(c.y, c.z));
  return ff_add(l, ff_add(r, make_float2(poly, 0.f)));
}

/* 2u - 1 as a pair: 24 bits, then the 29 below them. */
__device__ __forceinline__ float2 ff_signed(uint64_t w) {
  const int32_t top = (int32_t)(fi_hi32(w) ^ 0x80000000u);
  const uint32_t low = ((uint32_t)top & 0xffu) << 21 | ((uint32_t)(w >> 11) & 0x1fffffu);
  return ff_two((float)(top >> 8) * 0x1.0p-23f, (float)low * 0x1.0p-52f);
}

/* One try of the polar method on pairs.  q is good to 2^-46, so z is off
 * by less than 2^-46.5 / sqrt(1 - q) + 2^-40 + s 2^-49 (s = z / u), below
 * 2^-38 for q in [2^-12, 1 - 2^-12]; outside, FP64 decides. */
__device__ __forceinline__ int ff_polar(const FiTables* T, uint64_t w0, uint64_t w1, float2* z) {
  const float2 u = ff_signed(w0), v = ff_signed(w1);
  const float2 q = ff_add(ff_mul(u, u), ff_mul(v, v));
  if (q.x >= 1.0f + 0x1.0p-20f) return FI_REJECT;
  if (q.x > 1.0f - 0x1.0p-12f || q.x < 0x1.0p-12f) return FI_UNSURE;
  const float2 l = ff_log(T, q);
  *z = ff_mul(u, ff_sqrt(ff_div(make_float2(-2.0f * l.x, -2.0f * l.y), q)));
  return FI_OK;
}

/* Whether every value within 2^-34 relative of the pair v (v.x positive,
 * |v.y| at most half its last bit) rounds to the FP32 value v.x. */
__device__ __forceinline__ bool ff_sure(float2 v) {
  const uint32_t b = __float_as_uint(v.x);
  if (b < (40u << 23) || b >= (254u << 23) || (b & 0x7fffffu) == 0) return false;
  const float half = __uint_as_float((b & 0x7f800000u) - (24u << 23));
  return fabsf(v.y) < half - v.x * 0x1.0p-34f;
}

/* e^x for |x| < 60: x = (64 q + j) ln2/64 + r. */
__device__ __forceinline__ float2 ff_exp(const FiTables* T, float2 x) {
  const float n = rintf(x.x * 0x1.715476p+6f); /* 64 / ln 2 */
  /* ln2/64 in 13, 24 and 24 bits: n times the first part is exact */
  const float h = __fmaf_rn(-n, 0x1.62ep-7f, x.x);
  const float p = __fmul_rn(n, 0x1.0bfbe8p-21f);
  const float pe = __fmaf_rn(n, 0x1.0bfbe8p-21f, -p);
  float2 r = ff_two(h, -p);
  r = ff_fast2(r.x, __fadd_rn(r.y, __fsub_rn(__fsub_rn(x.y, pe), n * 0x1.cf79acp-46f)));
  const float t = r.x;
  float poly = __fmaf_rn(t, 0x1.555556p-5f, 0x1.555556p-3f);
  poly = __fmaf_rn(t, poly, 0.5f);
  poly = __fmul_rn(__fmul_rn(t, t), poly);
  const int k = (int)n, j = k & 63, e = (k - j) / 64;
  const float2 tab = T->exp_t[j];
  const float2 em1 = ff_add(r, make_float2(poly, 0.f));
  const float2 m = ff_add(tab, ff_mul(tab, em1));
  const float s = __uint_as_float((uint32_t)(127 + e) << 23);
  return make_float2(m.x * s, m.y * s);
}

/* -ln(1 - Phi(z)) from its series about the nearest of the table's points;
 * the terms from the cube on in FP32. */
__device__ __forceinline__ float2 ff_neg_log_sf(const FiTables* T, float2 z) {
  const int k = (int)rintf((z.x - FI_G_LO) * (float)FI_G_STEPS);
  const float z0 = FI_G_LO + (float)k * (1.0f / FI_G_STEPS);
  const float2 t = ff_fast2(__fsub_rn(z.x, z0), z.y);
  const float4 a = T->g[k][0], b = T->g[k][1], c = T->g[k][2];
  float p = __fmaf_rn(t.x, c.y, c.x);
  p = __fmaf_rn(t.x, p, b.w);
  p = __fmaf_rn(t.x, p, b.z);
  float2 s = ff_two(b.x, __fmul_rn(t.x, p));
  s.y = __fadd_rn(s.y, b.y);
  s = ff_add(ff_mul(s, t), make_float2(a.z, a.w));
  return ff_add(ff_mul(s, t), make_float2(a.x, a.y));
}

struct FiHet {
  uint64_t seed;
  int64_t capacity;
  float2 mu, sigma, rho, srho, scale;
  const FiTables* tab;
  float *risk, *inf;
};

/* Two normals a slot: the first block's two tries give both for 61.6% of
 * the slots; the rest keep the normal they have and take later blocks by
 * full warps.  Bound by integer (Philox) and FP32 issue; at 2.3e8 slots
 * timers and heterogeneity together took 687 ms in FP64. */
__global__ void __launch_bounds__(FI_THREADS) k_init_het_fast(FiHet A) {
  __shared__ FiTables T;
  __shared__ float4 s_z[FI_TILE]; /* z0, z1; NaN for unsure */
  __shared__ uint16_t s_open[FI_TILE];
  __shared__ int s_count;
  {
    const float4* src = reinterpret_cast<const float4*>(A.tab);
    float4* dst = reinterpret_cast<float4*>(&T);
    for (int k = threadIdx.x; k < (int)(sizeof(FiTables) / 16); k += FI_THREADS) dst[k] = src[k];
  }
  const float nan = __uint_as_float(0x7fc00000u);
  const int64_t tiles = (A.capacity + FI_TILE - 1) / FI_TILE;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t i0 = tile * FI_TILE;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    for (int o = threadIdx.x; o < FI_TILE; o += FI_THREADS) {
      if (i0 + o >= A.capacity) break;
      uint64_t c[4] = {(uint64_t)(i0 + o), 0, (uint64_t)LPG_P_INIT_HET << 32, 0};
      lpg_philox4x64_10(c, A.seed, LPG_KEY_TAG);
      float2 z0 = make_float2(0.f, 0.f), z1 = z0;
      const int a = ff_polar(&T, c[0], c[1], &z0);
      const int b = ff_polar(&T, c[2], c[3], &z1);
      float4 out = make_float4(z0.x, z0.y, z1.x, z1.y);
      if (a == FI_UNSURE || b == FI_UNSURE) {
        out.x = nan;
      } else if (a != FI_OK || b != FI_OK) {
        const int have = a == FI_OK || b == FI_OK;
        if (a != FI_OK) out = make_float4(z1.x, z1.y, 0.f, 0.f);
        s_open[fi_place(&s_count)] = (uint16_t)(o | have << 15);
      }
      s_z[o] = out;
    }
    __syncthreads();
    const int todo = s_count;
    for (int q = threadIdx.x; q < todo; q += FI_THREADS) {
      const int o = s_open[q] & 0x7fff;
      int have = s_open[q] >> 15;
      float4 out = s_z[o];
      for (int blk = 1; have < 2; ++blk) {
        uint64_t c[4] = {(uint64_t)(i0 + o), 0, (uint64_t)LPG_P_INIT_HET << 32, (uint64_t)blk};
        lpg_philox4x64_10(c, A.seed, LPG_KEY_TAG);
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          float2 z;
          const int a = have < 2 ? ff_polar(&T, c[2 * w], c[2 * w + 1], &z) : FI_REJECT;
          if (a == FI_UNSURE || blk > 64) {
            out.x = nan;
            have = 2;
          } else if (a == FI_OK) {
            if (have == 0) {
              out.x = z.x;
              out.y = z.y;
            } else {
              out.z = z.x;
              out.w = z.y;
            }
            ++have;
          }
        }
      }
      s_z[o] = out;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < FI_TILE; o += FI_THREADS) {
      const int64_t i = i0 + o;
      if (i >= A.capacity) break;
      const float4 zz = s_z[o];
      const float2 z0 = make_float2(zz.x, zz.y), z1 = make_float2(zz.z, zz.w);
      bool ok = zz.x == zz.x;
      float risk = 0.f, inf = 0.f;
      if (ok) {
        const float2 x = ff_add(A.mu, ff_mul(A.sigma, z0));
        const float2 zc = ff_add(ff_mul(A.rho, z0), ff_mul(A.srho, z1));
        ok = fabsf(x.x) < 60.0f && zc.x >= FI_G_LO && zc.x <= FI_G_HI;
        if (ok) {
          const float2 r = ff_exp(&T, x), g = ff_mul(A.scale, ff_neg_log_sf(&T, zc));
          ok = ff_sure(r) && ff_sure(g);
          risk = r.x;
          inf = g.x;
        }
      }
      A.risk[i] = ok ? risk : -1.0f; /* -1: for k_init_fix */
      A.inf[i] = inf;
    }
    __syncthreads();
  }
}

/* --- dates: the FP64 definitions' integers by integer arithmetic ------------- */
/* floor(u * span) as FP64 gives it, u = m 2^-53 and 0 <= span < 2^31: the
 * exact product's floor, unless the product lies so close below a whole
 * number (2^-21) that its rounding to 53 bits may reach it. */
__device__ __forceinline__ int64_t fi_scaled_floor(uint64_t m, int64_t span) {
  const uint64_t a = m << 11, lo = a * (uint64_t)span;
  if ((lo >> 43) == 0x1fffff || (uint64_t)span >> 31)
    return (int64_t)floor((double)m * 0x1.0p-53 * (double)span);
  return (int64_t)__umul64hi(a, (uint64_t)span);
}

/* The date tables of a CTA, in shared memory where they fit (FI_TABLE
 * entries), with guides: the first entry that a draw of the bucket can
 * reach, so that a search is one or two steps and not seven. */
#define FI_TABLE 256
#define FI_GUIDE 256
struct FiDates {
  const int64_t *cum, *km;
  const int32_t *lo, *hi;
  int32_t n_bins, km_len, km_max_year;
  int64_t s_cum[FI_TABLE], s_km[FI_TABLE];
  int32_t s_lo[FI_TABLE], s_hi[FI_TABLE];
  uint16_t age_guide[FI_GUIDE], km_guide[FI_GUIDE];
  float km_scale; /* buckets per death */
};

__device__ __forceinline__ int32_t fi_first_above(const int64_t* cum, int32_t n, int64_t v) {
  int32_t a = 0, b = n;
  while (a < b) {
    const int32_t m = (a + b) >> 1;
    if (cum[m] > v) b = m; else a = m + 1;
  }
  return a;
}

/* All threads of the CTA; the guides hold for tables of fewer than 65536
 * entries (start at entry 0 otherwise). */
__device__ __forceinline__ void fi_dates_load(FiDates& D, const int64_t* cum, const int32_t* lo, const int32_t* hi,
                                              int32_t n_bins, const int64_t* km, int32_t km_len, int32_t km_max_year) {
  const bool ages = cum != nullptr, deaths = km != nullptr;
  if (threadIdx.x == 0) {
    D.n_bins = n_bins;
    D.km_len = km_len;
    D.km_max_year = km_max_year;
    D.cum = n_bins <= FI_TABLE ? D.s_cum : cum;
    D.lo = n_bins <= FI_TABLE ? D.s_lo : lo;
    D.hi = n_bins <= FI_TABLE ? D.s_hi : hi;
    D.km = km_len <= FI_TABLE ? D.s_km : km;
  }
  if (ages && n_bins <= FI_TABLE)
    for (int q = threadIdx.x; q < n_bins; q += blockDim.x) {
      D.s_cum[q] = cum[q];
      D.s_lo[q] = lo[q];
      D.s_hi[q] = hi[q];
    }
  if (deaths && km_len <= FI_TABLE)
    for (int q = threadIdx.x; q < km_len; q += blockDim.x) D.s_km[q] = km[q];
  __syncthreads();
  const int32_t top = km_max_year < km_len - 1 ? km_max_year : km_len - 1;
  for (int b = threadIdx.x; b < FI_GUIDE; b += blockDim.x) {
    if (ages) {
      /* bucket b: the uniform's top 8 bits */
      const uint64_t v = lpg_scale_target((uint64_t)b << 45, (uint64_t)cum[n_bins - 1]);
      D.age_guide[b] = n_bins < 65536 ? (uint16_t)fi_first_above(D.cum, n_bins - 1, (int64_t)v) : 0;
    }
    if (deaths) {
      /* bucket b: draws from (b - 1) / 256 of the total on, a bucket's slack for the FP32 scaling */
      const int64_t total = top >= 0 ? km[top] : 0;
      const int64_t from = b > 0 && total > 0 ? (int64_t)((double)total * (b - 1) / FI_GUIDE) : INT64_MIN;
      D.km_guide[b] = top >= 0 && km_len < 65536 ? (uint16_t)fi_first_above(D.km, top + 1, from) : 0;
      if (b == 0) D.km_scale = total > 0 ? (float)FI_GUIDE / (float)total : 0.0f;
    }
  }
  __syncthreads();
}

/* lpg_init_age */
__device__ __forceinline__ int32_t fi_age(const FiDates& D, uint64_t seed, uint64_t slot) {
  uint64_t w[4] = {slot, 0, (uint64_t)LPG_P_INIT_AGE << 32, 0};
  lpg_philox4x64_10(w, seed, LPG_KEY_TAG);
  const uint64_t m = w[0] >> 11;
  const int64_t v = (int64_t)lpg_scale_target(m, (uint64_t)D.cum[D.n_bins - 1]);
  int32_t a = D.age_guide[m >> 45]; /* first bin with cum > v */
  while (a < D.n_bins - 1 && D.cum[a] <= v) ++a;
  const int32_t age = D.lo[a] + (int32_t)fi_scaled_floor(w[1] >> 11, D.hi[a] - D.lo[a]);
  return age < 1 ? 1 : age;
}

/* lpg_km_age_at_death from the 53-bit integers of its uniforms */
__device__ __forceinline__ int32_t fi_age_at_death(const FiDates& D, int64_t age_days, uint64_t m0, uint64_t m1) {
  const int32_t top = D.km_max_year < D.km_len - 1 ? D.km_max_year : D.km_len - 1;
  int64_t years = age_days >> 30 ? age_days / 365 : (int64_t)((int32_t)age_days / 365);
  if (years > top) years = top;
  const int64_t lower = years > 0 ? D.km[years - 1] : 0;
  const int64_t total = D.km[top];
  const int64_t span = total - lower > 0 ? total - lower : 0;
  int64_t y = top;
  if (span > 0) {
    const int64_t draw = lower + fi_scaled_floor(m0, span);
    const float at = (float)draw * D.km_scale;
    int32_t a = D.km_guide[at <= 0.0f ? 0 : at < (float)(FI_GUIDE - 1) ? (int)at : FI_GUIDE - 1];
    while (a <= top && D.km[a] <= draw) ++a; /* first index with cum > draw, top + 1 if none */
    y = a > years ? a : years;
    if (y > top) y = top;
  }
  const int64_t day_lo = y == years ? age_days : y * 365;
  int64_t day_hi = (y + 1) * 365;
  if (day_hi < day_lo + 1) day_hi = day_lo + 1;
  return (int32_t)(day_lo + fi_scaled_floor(m1, day_hi - day_lo));
}

/* lpg_init_ri: dob + (42 + 56 u) truncated.  The FP64 sum is within 2^-20 of
 * the exact one; a fraction that close to a whole day is left to FP64. */
__device__ __forceinline__ int16_t fi_ri(uint64_t seed, uint64_t slot, int32_t dob) {
  const uint64_t m = lpg_u53(seed, LPG_P_INIT_RI, 0, slot, 0, 0);
  const uint64_t days = 56 * m; /* 53 fraction bits */
  const uint32_t f = (uint32_t)(days >> 21) /* 32 fraction bits */;
  const int64_t v = (int64_t)dob + 42 + (int64_t)(days >> 53);
  if (f < 0x2000u || f > 0xffffdfffu || v > 0x7ffffff0) return lpg_init_ri(seed, slot, dob);
  const int32_t d = (int32_t)(v < 0 ? v + 1 : v); /* towards zero, never whole */
  return (int16_t)(uint16_t)(uint32_t)d;
}

/* --- the slots left to FP64 -------------------------------------------------- */
struct FiExact {
  uint64_t seed;
  int64_t capacity;
  int32_t k_exp, k_inf, k_par;
  double e1, e2, i1, i2, p1, p2;
  double mu, sigma, rho, srho, scale;
  lpg_columns c;
};

/* Marked slots of a tile are listed first, so that the long FP64 chains run
 * in full warps (a tile of 16384 slots holds 30 to 80 of them). */
template <bool HET>
__global__ void __launch_bounds__(FI_THREADS) k_init_fix(FiExact A) {
  __shared__ uint16_t s_list[FI_FIX_TILE];
  __shared__ int s_count;
  const int64_t tiles = (A.capacity + FI_FIX_TILE - 1) / FI_FIX_TILE;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t i0 = tile * FI_FIX_TILE;
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    const int n = (int)(A.capacity - i0 < FI_FIX_TILE ? A.capacity - i0 : FI_FIX_TILE);
#pragma unroll 8
    for (int o = threadIdx.x; o < n; o += FI_THREADS) {
      const bool marked = HET ? A.c.acq_risk_multiplier[i0 + o] == -1.0f : A.c.infection_timer[i0 + o] == -1;
      if (marked) s_list[fi_place(&s_count)] = (uint16_t)o;
    }
    __syncthreads();
    const int todo = s_count;
    for (int q = threadIdx.x; q < todo; q += FI_THREADS) {
      const int64_t i = i0 + s_list[q];
      if (HET)
        lpg_init_het(A.seed, (uint64_t)i, 1, A.mu, A.sigma, A.rho, A.srho, A.scale, &A.c.acq_risk_multiplier[i],
                     &A.c.daily_infectivity[i]);
      else
        lpg_init_timers(A.seed, (uint64_t)i, A.k_exp, A.e1, A.e2, A.k_inf, A.i1, A.i2, A.k_par, A.p1, A.p2,
                        &A.c.exposure_timer[i], &A.c.infection_timer[i], &A.c.paralysis_timer[i]);
    }
    __syncthreads();
  }
}

/* --- host side ------------------------------------------------------------- */
/* A timer distribution's FP32 form; false where there is none (the FP64
 * kernel then fills the timers): kinds and ranges in which the error bounds
 * above hold and an unsure draw is rare.  thr receives the Poisson
 * thresholds: u > f_k exactly when the 53-bit integer m = u 2^53 exceeds
 * floor(f_k 2^53), f_k the running sums as lpg_poisson forms them. */
inline bool fi_dist_of(const lpg_dist& d, FiDist* out, std::vector<uint64_t>* thr) {
  *out = FiDist{};
  out->kind = d.kind;
  switch (d.kind) {
    case LPG_DIST_CONSTANT:
      out->value = (float)d.p1;
      return d.p1 >= 0.0 && d.p1 < 1048576.0 && (double)out->value == d.p1;
    case LPG_DIST_GAMMA: {
      if (!(d.p1 >= 1.0 && d.p1 <= 64.0 && d.p2 > 0.0 && d.p2 * d.p1 < 4096.0)) return false;
      double gd, gc;
      lpg_gamma_consts(d.p1, &gd, &gc);
      out->d = (float)gd;
      out->c = (float)gc;
      out->scale = (float)(gd * d.p2);
      return true;
    }
    case LPG_DIST_LOGNORMAL: {
      if (!(d.p1 > 0.0 && d.p1 < 4096.0 && d.p2 >= 0.01 * d.p1 && d.p2 <= 8.0 * d.p1)) return false;
      out->mu = (float)std::log(d.p1 * d.p1 / std::sqrt(d.p2 * d.p2 + d.p1 * d.p1));
      out->sg = (float)std::sqrt(std::log(d.p2 * d.p2 / (d.p1 * d.p1) + 1.0));
      return std::fabs(out->mu) < 16.0f;
    }
    case LPG_DIST_POISSON: {
      if (!(d.p1 > 0.0 && d.p1 < 10.0)) return false;
      double p = lpg_exp(-d.p1), f = p;
      for (int64_t x = 0; x < 64; ++x) {
        if (x > 0) {
          p = (p * d.p1) * lpg_recip_small(x);
          f = f + p;
        }
        thr->push_back(f >= 1.0 ? 1ULL << 53 : (uint64_t)(f * 9007199254740992.0));
        if (f >= 1.0) break;
      }
      return true;
    }
    default: return false;
  }
}

inline float2 fi_pair(double x) {
  const float hi = (float)x;
  return make_float2(hi, (float)(x - (double)hi));
}

/* The tables, in double precision from the C library's log, exp2 and erfc.
 * The series of g = -ln(1 - Phi) about z: g' = h, the hazard phi/(1 - Phi),
 * and h' = h^2 - z h gives every further coefficient. */
inline FiTables* fi_tables() {
  FiTables* T = new FiTables();
  for (int j = 0; j < FI_LOG_N; ++j) {
    const double F = j < 64 ? 1.0 + j / 128.0 : (1.0 + j / 128.0) / 2.0;
    const float c = (float)(1.0 / F);
    const float2 l = fi_pair(-std::log((double)c));
    T->log_c[j] = make_float4(c, l.x, l.y, 0.f);
  }
  for (int j = 0; j < FI_EXP_N; ++j) T->exp_t[j] = fi_pair(std::exp2(j / 64.0));
  for (int k = 0; k < FI_G_N; ++k) {
    const double z = (double)FI_G_LO + k / (double)FI_G_STEPS;
    const double tail = 0.5 * std::erfc(std::fabs(z) * LPG_SQRT1_2); /* P(Z > |z|) */
    const double sf = z >= 0.0 ? tail : 1.0 - tail;
    double h[6], g[7];
    g[0] = z >= 0.0 ? -std::log(sf) : -std::log1p(-tail);
    h[0] = std::exp(-0.5 * z * z) / std::sqrt(2.0 * LPG_PI) / sf;
    for (int n = 0; n < 5; ++n) {
      double s = -z * h[n] - (n ? h[n - 1] : 0.0);
      for (int i = 0; i <= n; ++i) s += h[i] * h[n - i];
      h[n + 1] = s / (n + 1);
    }
    for (int n = 0; n < 6; ++n) g[n + 1] = h[n] / (n + 1);
    const float2 c0 = fi_pair(g[0]), c1 = fi_pair(g[1]), c2 = fi_pair(g[2]);
    T->g[k][0] = make_float4(c0.x, c0.y, c1.x, c1.y);
    T->g[k][1] = make_float4(c2.x, c2.y, (float)g[3], (float)g[4]);
    T->g[k][2] = make_float4((float)g[5], (float)g[6], 0.f, 0.f);
  }
  return T;
}

#endif /* LPG_INIT_FAST_CUH */
