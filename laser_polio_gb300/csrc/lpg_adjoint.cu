/*
 * lpg_adjoint.cu — expected incidence of a tick range and its
 * vector-Jacobian product (lpg_incidence_plan_* and lpg_expected_incidence
 * in lpg.h).
 *
 * With the agent state held fixed, the transmission step's node-level part
 * (model.py:1315-1363) maps the replayed aggregates of each tick t — the
 * susceptibles' risk sum srisk[t,n], the pre-mixing infectivity
 * beta[t,n,s], the population pop[t,n] — to the expected exposures
 *
 *   N        = rownorm(gravity(p, d, k, a, b, c) / (sum p)^c, m)       (model.py:1250-1258)
 *   u[t,n,s] = beta[t,n,s] (1 - sum_k N[n,k]) + sum_i N[i,n] beta[t,i,s]
 *   seas[t]  = 1 + amp cos(2 pi (doy[t] - peak) / year[t])             (utils.py:589-625)
 *   r        = u seas[t] r0s[n] R / max(pop[t,n], 1)
 *   lam[t,n] = srisk[t,n] sum_s (1 - exp(-r))
 *
 * where R scales every agent's infectivity (R0 over the R0 the aggregates
 * were recorded at).  Given dL/dlam, the reverse pass returns dL/dR, dL/damp,
 * dL/dpeak, dL/dr0s, dL/dN and dL/d(k, a, b, c) through the row
 * normalisation (a row whose sum exceeds m is scaled down to m) and the
 * gravity flows k p_i^a p_j^b / d_ij^c (zero diagonal).  With a target
 * curve the plan also forms the calibration loss
 * L = sum (log1p(lam) - log1p(target))^2 and its dL/dlam on the device.
 *
 * Layout in HBM: a plan keeps the aggregates resident — srisk and
 * max(pop, 1) [T][G]; beta as [T][S][G] (strain-major per tick, so that the
 * (t, s) rows of the mixing product and every elementwise pass read G
 * consecutive doubles); u the same way, and dL/du in its place; log(dist),
 * log2(dist) and the flows and their gradients [G][G]; log(pops) [G].  The
 * sliced products' digits take 48 bytes an element of beta up to INC_DIGITS
 * elements, and no more than for those above: 200 MB.
 *
 * Arithmetic: double precision throughout, most of it without the FP64 unit.
 * GB300 issues about two FP64 FMAs per clock per SM, 128 FP32 or integer
 * operations, and 8192 bf16 tensor FMAs.
 *   - The two contractions, u = beta N per (t, s) row and dL/dN = beta^T
 *     dL/du, both (T S) x G x G, run on the tensor cores by exact slicing
 *     (lpg_ozaki.cuh).  beta's slices are formed once per plan (by
 *     columns with the target or at the first gradient), N's and dL/du's each
 *     evaluation.  An element that is small beside its row's and
 *     column's scales is formed again from the FP64 operands, so that each
 *     element is good to 2^-45 of its own summed terms (four deviations; the
 *     FP32 pairs used where many are small: rms).
 *   - Contractions too small for that are summed in FP64 where their results
 *     are used, with no launch of their own.
 *   - exp and log1p run in 64-bit integer arithmetic (lpg_ixmath.cuh).
 * The sums use atomics, so results agree with a sequential FP64 evaluation
 * to rounding, not bit for bit.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "lpg.h"
#include "lpg_ixmath.cuh"
#include "lpg_ozaki.cuh"

/* Per-host-thread error text of the standalone ops (lpg_ops.cu). */
int lpg_ops_fail(int code, const char* fmt, ...);

namespace {

constexpr double kTwoPi = 6.283185307179586476925286766559;
#define INC_THREADS 256
#define INC_MAX_SPLIT 8 /* depth slices of a sliced product */
#define INC_MAX_ROWS (65535 * 32)
#define INC_SMALL_NODES 128
#define INC_SMALL_TERMS 4000000 /* T S G^2 */
#define INC_DIGITS (1 << 22)    /* elements of beta whose digits a plan keeps (16 bytes each) */

enum { PH_NETWORK, PH_MIX, PH_FORWARD, PH_BACKWARD, PH_FLOWS, PH_NETWORK_GRAD, PH_COUNT };
const char* const kPhaseNames[PH_COUNT] = {"k_inc_network", "k_inc_gemm_mix", "k_inc_forward",
                                           "k_inc_backward", "k_inc_gemm_flows", "k_inc_network_grad"};

struct IncScalars {
  double R, amp, peak;
};

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

/* The sum over the CTA (whole warps, at most 32), in every thread.  An FP64
 * addition holds the pipe for 16 cycles a warp, so only the first warp adds
 * the warps' sums. */
__device__ __forceinline__ double block_sum(double v, double* s_part) {
  const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    double r = lane < warps ? s_part[lane] : 0.0;
    for (int o = 1; o < warps; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    if (lane == 0) s_part[0] = r;
  }
  __syncthreads();
  return s_part[0];
}

#define INC_LOG2_NONE INT64_MIN /* log2 of 0 or infinity */

/* log2 x with 52 fraction bits. */
__device__ __forceinline__ int64_t inc_log2(double x) {
  if (!(x > 0.0) || isinf(x)) return INC_LOG2_NONE;
  int e;
  const double m = frexp(x, &e); /* [1/2, 1): log2 m to 2^-53 absolute */
  return ((int64_t)e << 52) + __double2ll_rn(log2(m) * 0x1p52);
}

/* log(pops), log2(pops) [G]; log(dist), log2(dist) [G][G] (the diagonal is
 * never read); max(pop, 1) and log1p(target) [T][G]: once per plan.  The
 * distances' log2 in integers: one FP64 logarithm a cell, not two (774 nodes:
 * 1.03 ms with both, about half now; ln in integers would be 0.9 ulp off
 * where CUDA's is 0.54). */
__global__ void __launch_bounds__(INC_THREADS)
    k_inc_logs(const IxTables* tab, int G, size_t TG, const double* pops, const double* dist, double* logp,
               double* logd, int64_t* lp2, int64_t* ld2, const double* pop, double* popc, double* target) {
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < (size_t)G * G) {
    const double x = dist[idx];
    logd[idx] = log(x);
    ld2[idx] = x >= 0x1p-1022 && x < HUGE_VAL ? ix_log2(tab, x) : inc_log2(x);
  }
  if (idx < (size_t)G) {
    logp[idx] = log(pops[idx]);
    lp2[idx] = inc_log2(pops[idx]);
  }
  if (idx < TG) {
    popc[idx] = fmax(pop[idx], 1.0);
    if (target) target[idx] = log1p(target[idx]);
  }
}

/* a c 2^-56, rounded: a with 52 fraction bits times c with 56. */
__device__ __forceinline__ int64_t inc_mul56(int64_t a, int64_t c) {
  const int64_t hi = __mul64hi(a, c);
  const uint64_t lo = (uint64_t)a * (uint64_t)c;
  return (int64_t)((uint64_t)hi << 8 | lo >> 56) + (int64_t)(lo >> 55 & 1);
}

/* The gravity parameters of an evaluation: kP = k / P^c; a, b, c also with
 * 56 fraction bits.  integer: every exponent stays within the fixed-point
 * range (the host's check), so that the flows are formed in integers. */
struct IncGravity {
  double a, b, c, kP, max_frac;
  int64_t a56, b56, c56;
  int integer;
};

/* kP p^a */
__device__ __forceinline__ double inc_row_scale(const IxTables* T, const IncGravity& V, double p, int64_t l2) {
  if (!V.integer || (l2 == INC_LOG2_NONE && V.a != 0.0)) return V.kP * pow(p, V.a);
  if (V.a == 0.0) return V.kP;
  const int64_t E = inc_mul56(l2, V.a56);
  return V.kP * ix_double(ix_exp2_frac(T, (uint64_t)E << 12), (int)(E >> 52));
}

/* Blocks [0, G): one network row i each — the scaled gravity flows
 * G[i,j] = k p_i^a p_j^b / d_ij^c / P^c (zero diagonal; non-finite
 * values are 0), formed as k p_i^a 2^(b log2 p_j - c log2 d_ij) / P^c with
 * the 0^0 = 1 convention kept, their sum rs[i], the factor fac[i] that scales
 * the row down to max_frac when rs[i] exceeds it (else 1), and the normalised
 * row's sum; for the small sums also the normalised row N[i,j].
 * Blocks [G, G + ceil(T/32)): the seasonal factor of each tick and its
 * derivatives with respect to amp and peak.
 * Bound by integer issue (about 110 instructions an element, one FP64
 * addition); with the FP64 library's pow and exp 774 nodes took 94 us. */
template <bool SMALL>
__global__ void __launch_bounds__(INC_THREADS)
    k_inc_network(int G, int T, const IxTables* __restrict__ tab, const double* pops, const double* logp,
                  const double* logd, const int64_t* lp2, const int64_t* __restrict__ ld2, IncGravity V, double* Gm,
                  double* N, double* rs, double* rsN, double* fac, const double* doy, const double* year,
                  IncScalars sc, double* seas) {
  __shared__ double s_part[INC_THREADS / 32], s_kpa;
  if ((int)blockIdx.x >= G) {
    /* a warp a block: the FP64 sine, cosine and divisions of 256 ticks on one SM would outlast the rows */
    const int t = (blockIdx.x - G) * 32 + threadIdx.x;
    if (threadIdx.x < 32 && t < T) {
      const double ang = kTwoPi * (doy[t] - sc.peak) / year[t];
      double sa, ca;
      sincos(ang, &sa, &ca);
      seas[t] = 1.0 + sc.amp * ca;
      seas[T + t] = ca;                                 /* d seas / d amp */
      seas[2 * T + t] = sc.amp * sa * kTwoPi / year[t]; /* d seas / d peak */
    }
    return;
  }
  const int i = blockIdx.x;
  if (threadIdx.x == 0) s_kpa = inc_row_scale(tab, V, pops[i], lp2[i]);
  __syncthreads();
  const double kpa = s_kpa;
  const uint64_t kb = (uint64_t)__double_as_longlong(kpa);
  const int kx = (int)(kb >> 52 & 0x7ff);
  const uint64_t km = ((kb & 0xfffffffffffffULL) | 1ULL << 52) << 11;
  const bool integer = V.integer && kx > 0 && kx < 0x7ff;
  double sum = 0.0;
  for (int j = threadIdx.x; j < G; j += blockDim.x) {
    double v = 0.0;
    if (j != i) {
      if (integer) {
        const int64_t l = lp2[j], d = ld2[(size_t)i * G + j];
        if ((l != INC_LOG2_NONE || V.b == 0.0) && (d != INC_LOG2_NONE || V.c == 0.0)) {
          const int64_t E = (V.b == 0.0 ? 0 : inc_mul56(l, V.b56)) - (V.c == 0.0 ? 0 : inc_mul56(d, V.c56));
          uint64_t m = __umul64hi(ix_exp2_frac(tab, (uint64_t)E << 12), km);
          int n = (int)(E >> 52) + kx - 1022;
          if (!(m >> 63)) {
            m <<= 1;
            n -= 1;
          }
          if (n >= -1022 && n <= 1022) v = __longlong_as_double(__double_as_longlong(ix_double(m, n)) | (long long)(kb & 1ULL << 63));
        }
      } else {
        const double x = (V.b == 0.0 ? 0.0 : V.b * logp[j]) - (V.c == 0.0 ? 0.0 : V.c * logd[(size_t)i * G + j]);
        v = kpa * exp(x);
        if (!isfinite(v)) v = 0.0;
      }
    }
    Gm[(size_t)i * G + j] = v;
    sum += v;
  }
  const double r = block_sum(sum, s_part);
  const bool cap = r > V.max_frac;
  const double f = cap ? V.max_frac / r : 1.0;
  double rn = r;
  if (SMALL || cap) {
    double sumN = 0.0;
    for (int j = threadIdx.x; j < G; j += blockDim.x) {
      const double v = Gm[(size_t)i * G + j]; /* written by this thread above */
      const double nv = cap ? v * f : v;
      if (SMALL) N[(size_t)i * G + j] = nv;
      sumN += nv;
    }
    rn = block_sum(sumN, s_part);
  }
  if (threadIdx.x == 0) {
    rs[i] = r;
    rsN[i] = rn;
    fac[i] = f;
  }
}

__device__ __forceinline__ double inc_exp_neg(const IxTables* tab, double x) {
  return ix_below(x, 700.0) ? ix_exp_neg(tab, x) : exp(-x);
}

__device__ __forceinline__ double inc_log1p(const IxTables* tab, double y) {
  return ix_below(y, 0x1p60) && !ix_below(y, 0x1p-5) ? ix_log1p(tab, y) : log1p(y);
}

struct IncStep {
  int T, G, S;
  const double *srisk, *beta, *popc, *seas, *r0s, *rsN, *ltarget, *g_in;
  const double* u; /* the mixing product, or */
  const double* N; /* the normalised network (small sums) */
  double R;
  double *lam, *loss; /* lam may be null */
  double* gu; /* dL/du */
  unsigned long long* max_gu;
  double *g_r0s, *g_w;
  int grad;
};

/* TC ticks of one node a thread: the mixing's diagonal term, the rates,
 * lam, with a target the loss term and dL/dlam, and with grad the reverse
 * pass of the same cells: dL/du, its column maxima, the r0s gradient, and
 * w[t] = sum_n dL/dq / popc r0s, from which the last kernel forms the
 * gradients of R, amp and peak.  Forward and reverse share the rates and
 * exponentials in registers (they were two kernels and 2 T S G doubles
 * between them).  Bound by FP64 issue: about 32 operations a cell, the
 * exponentials and logarithms in integers (774 nodes, 365 ticks, 3 strains:
 * 185 us before). */
template <bool SMALL, int TC>
__global__ void __launch_bounds__(128, SMALL ? 4 : 6) k_inc_step(const IxTables* __restrict__ tab, IncStep A) {
  __shared__ double s_loss[4];
  const int n = blockIdx.x * 128 + threadIdx.x, t0 = blockIdx.y * TC, lane = threadIdx.x & 31;
  const int T = A.T, G = A.G, S = A.S;
  const bool in = n < G;
  const double keep = in ? 1.0 - A.rsN[n] : 0.0, r0 = in ? A.r0s[n] : 0.0;
  double loss = 0.0, acc_r0 = 0.0;
  unsigned long long mx = 0;
  double w[TC];
#pragma unroll
  for (int i = 0; i < TC; ++i) {
    w[i] = 0.0;
    const int t = t0 + i;
    if (!in || t >= T) continue;
    const size_t idx = (size_t)t * G + n;
    const double st = A.seas[t];
    const IxDivisor popc(A.popc[idx]);
    const double q = popc.of(st * r0 * A.R);
    double uu[LPG_MAX_STRAINS], ex[LPG_MAX_STRAINS], l = 0.0, mix[LPG_MAX_STRAINS] = {0.0, 0.0, 0.0, 0.0};
    if (SMALL) {
      const double* b = A.beta + (size_t)t * S * G;
#pragma unroll 8
      for (int j = 0; j < G; ++j) {
        const double m = A.N[(size_t)j * G + n];
#pragma unroll
        for (int s = 0; s < LPG_MAX_STRAINS; ++s)
          if (s < S) mix[s] = __fma_rn(b[s * G + j], m, mix[s]);
      }
    }
#pragma unroll
    for (int s = 0; s < LPG_MAX_STRAINS; ++s) {
      uu[s] = ex[s] = 0.0;
      if (s >= S) continue;
      const size_t k = ((size_t)t * S + s) * G + n;
      uu[s] = __fma_rn(A.beta[k], keep, SMALL ? mix[s] : A.u[k]);
      ex[s] = inc_exp_neg(tab, uu[s] * q);
      l += 1.0 - ex[s];
    }
    const double sr = A.srisk[idx], lv = sr * l;
    if (A.lam) A.lam[idx] = lv;
    double g = 0.0;
    if (A.ltarget) {
      const double r = inc_log1p(tab, lv) - A.ltarget[idx];
      g = IxDivisor(1.0 + lv).of(2.0 * r);
      loss = __fma_rn(r, r, loss);
    }
    if (!A.grad) continue;
    if (A.g_in) g = A.g_in[idx];
    const double gs = g * sr;
    double gq = 0.0;
#pragma unroll
    for (int s = 0; s < LPG_MAX_STRAINS; ++s) {
      if (s >= S) continue;
      const size_t k = ((size_t)t * S + s) * G + n;
      const double gr = gs * ex[s], gu = gr * q;
      A.gu[k] = gu;
      const unsigned long long b = oz_abs_bits(gu);
      mx = b > mx ? b : mx;
      gq = __fma_rn(gr, uu[s], gq);
    }
    const double gp = popc.of(gq);
    w[i] = gp * r0;
    acc_r0 = __fma_rn(gp * st, A.R, acc_r0);
  }
  if (A.grad) {
    if (in) {
      atomicAdd(&A.g_r0s[n], acc_r0);
      if (!SMALL) atomicMax(&A.max_gu[n], mx);
    }
#pragma unroll
    for (int i = 0; i < TC; ++i) {
      const double v = warp_sum(w[i]);
      if (lane == 0 && t0 + i < T) atomicAdd(&A.g_w[t0 + i], v);
    }
  }
  if (A.ltarget) { /* uniform over the grid */
    loss = warp_sum(loss);
    if (lane == 0) s_loss[threadIdx.x >> 5] = loss;
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(A.loss, (s_loss[0] + s_loss[1]) + (s_loss[2] + s_loss[3]));
  }
}

/* The last block: dL/dR, dL/damp and dL/dpeak from w[t].  The others take
 * rows a in turn — C[a][b] of the flows product, or with SMALL the sum over
 * (t, s) formed here, dL/dN[a][b] = C[a][b] - C[a][a] (zero on the diagonal), then dL/dG
 * through the row normalisation and the contributions to dL/dk, dL/da, dL/db,
 * dL/dc, kept per thread over the CTA's rows; dL/dN is written when asked
 * for.  Bound by FP64 issue: five operations an element and two a row and
 * thread (4000 nodes: 616 us with a reduction and two passes a row). */
template <bool SMALL>
__global__ void __launch_bounds__(INC_THREADS, SMALL ? 2 : 5)
    k_inc_network_grad(int G, int T, int TS, const double* C, const double* beta, const double* gu, const double* Gm, const double* rs,
                       const double* fac, const double* logp, const double* logd, double k, double logP,
                       double* gN, double* g_theta, const double* seas, const double* g_w, double R, double* g_seas) {
  __shared__ double s_part[INC_THREADS / 32];
  const int rows = gridDim.x - 1;
  if ((int)blockIdx.x == rows) {
    double gR = 0.0, ga = 0.0, gp = 0.0;
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
      gR = __fma_rn(g_w[t], seas[t], gR);
      ga = __fma_rn(g_w[t] * R, seas[T + t], ga);
      gp = __fma_rn(g_w[t] * R, seas[2 * T + t], gp);
    }
    gR = block_sum(gR, s_part);
    ga = block_sum(ga, s_part);
    gp = block_sum(gp, s_part);
    if (threadIdx.x == 0) {
      g_seas[0] = gR;
      g_seas[1] = ga;
      g_seas[2] = gp;
    }
    return;
  }
  extern __shared__ double s_flow[]; /* the small sums: partial rows [slices][G] */
  auto nonzero = [](double x) { return ((uint64_t)__double_as_longlong(x) << 1) != 0; };
  double wk = 0.0, wa = 0.0, wb = 0.0, wc = 0.0;
  for (int a = blockIdx.x; a < G; a += rows) {
    const size_t row = (size_t)a * G;
    if (SMALL) {
      /* row a of beta^T dL/du: the depth cut over groups of threads, one column a thread */
      const int width = (G + 31) / 32 * 32 < INC_THREADS ? (G + 31) / 32 * 32 : INC_THREADS;
      const int slices = INC_THREADS / width, sl = threadIdx.x / width;
      const int per = (TS + slices - 1) / slices, k1 = min(TS, (sl + 1) * per);
      if (sl < slices)
        for (int b = threadIdx.x % width; b < G; b += width) {
          double c = 0.0;
#pragma unroll 8
          for (int k = sl * per; k < k1; ++k) c = __fma_rn(beta[(size_t)k * G + a], gu[(size_t)k * G + b], c);
          s_flow[sl * G + b] = c;
        }
      __syncthreads();
      for (int b = threadIdx.x; b < G; b += blockDim.x) {
        double c = s_flow[b];
        for (int q = 1; q < slices; ++q) c += s_flow[q * G + b];
        s_flow[b] = c;
      }
      __syncthreads();
    }
    auto flow = [&](int b) { return SMALL ? s_flow[b] : C[row + b]; };
    const double diag = flow(a), f = fac[a];
    const bool cap = f != 1.0;
    double shift = 0.0; /* a capped row's coupling: sum of dL/dN G over the row, by its sum */
    if (cap) {
      double cpl = 0.0;
      for (int b = threadIdx.x; b < G; b += blockDim.x)
        cpl = __fma_rn(b == a ? 0.0 : flow(b) - diag, Gm[row + b], cpl);
      shift = block_sum(cpl, s_part) / rs[a];
    }
    double wr = 0.0;
#pragma unroll 4
    for (int b = threadIdx.x; b < G; b += blockDim.x) {
      double gn = b == a ? 0.0 : flow(b) - diag;
      if (gN) gN[row + b] = gn;
      if (cap) gn = f * (gn - shift);
      const double w = b == a ? 0.0 : gn * Gm[row + b];
      if (nonzero(w)) { /* not a zero flow, whose logs may be infinite */
        wr += w;
        wb = __fma_rn(w, logp[b], wb);
        wc = __fma_rn(w, logd[row + b], wc);
      }
    }
    if (nonzero(wr)) {
      wk += wr;
      wa = __fma_rn(wr, logp[a], wa);
    }
    if (SMALL) __syncthreads(); /* the row is read before the next one is summed */
  }
  wk = block_sum(wk, s_part);
  wa = block_sum(wa, s_part);
  wb = block_sum(wb, s_part);
  wc = block_sum(wc, s_part);
  if (threadIdx.x == 0) {
    atomicAdd(&g_theta[0], wk / k);
    atomicAdd(&g_theta[1], wa);
    atomicAdd(&g_theta[2], wb);
    atomicAdd(&g_theta[3], -wc - wk * logP);
  }
}

}  // namespace

enum { SC_LOSS = 0, SC_R = 1, SC_THETA = 4, SC_ERR = 8, SC_LIST = 9, SC_N = 16 }; /* SC_LIST: two counts */

struct lpg_incidence_plan {
  int T = 0, G = 0, S = 0;
  int nsm = 0;
  cudaStream_t st = nullptr;
  bool own_stream = false;
  double P = 0.0, logP = 0.0;
  double max_lp2 = 0.0, max_ld2 = 0.0; /* largest finite |log2 pops|, |log2 dist| */
  bool small = false;                  /* the contractions summed in FP64 where they are used */
  /* resident inputs */
  double *srisk = nullptr, *beta = nullptr, *popc = nullptr, *doy = nullptr, *year = nullptr, *pops = nullptr,
         *logp = nullptr, *logd = nullptr, *target = nullptr; /* target: its log1p */
  int64_t *lp2 = nullptr, *ld2 = nullptr;
  IxTables* tab = nullptr;
  /* per evaluation */
  double *r0s = nullptr, *seas = nullptr, *Gm = nullptr, *rs = nullptr, *rsN = nullptr, *fac = nullptr,
         *u = nullptr, *lam = nullptr, *g = nullptr, *C = nullptr, *gN = nullptr;
  /* cleared each evaluation, one block: sums [SC_N], gr0s [G], w [T], column maxima of N and dL/du [G], their sums
   * of squares [G] */
  double *sums = nullptr, *gr0s = nullptr, *gw = nullptr;
  unsigned long long *max_n = nullptr, *max_gu = nullptr;
  uint32_t *sq_n = nullptr, *sq_gu = nullptr;
  size_t clear_bytes = 0;
  double *N = nullptr, *gu = nullptr; /* gu of the sliced products: in u's place */
  /* the sliced products: digits, row and column maxima and sums of squares, tensor maps.  Digits of row_cap rows
   * or dep_cap depths of beta at a time: all of them, kept, up to INC_DIGITS elements; above, a part after another in
   * every evaluation.  n_cols and C share their memory (the
   * mixing is done with the one before the flows write the other), gu_cols and the list theirs. */
  int row_cap = 0, dep_cap = 0;
  bool rows_ready = false, cols_ready = false, bc_ready = false;
  int polls = OZ_WAIT_POLLS, stall = -1; /* lpg_test_stall_products */
  uint32_t *b_rows = nullptr, *b_cols = nullptr, *n_cols = nullptr, *gu_cols = nullptr;
  unsigned long long *max_br = nullptr, *max_bc = nullptr;
  uint32_t *sq_br = nullptr, *sq_bc = nullptr;
  unsigned long long* list_n = nullptr; /* two of the sums */
  CUtensorMap map_b{}, map_n{}, map_bt{}, map_gu{};
  double* host = nullptr; /* pinned: sums and gr0s [SC_N + G], then r0s [G] */
  /* profiling */
  bool prof = false;
  cudaEvent_t ev[PH_COUNT + 1] = {};
  double ms[PH_COUNT] = {};
  int64_t evals[PH_COUNT] = {};
};

namespace {

int plan_cuda(cudaError_t e, const char* what) {
  return e == cudaSuccess ? LPG_OK : lpg_ops_fail(LPG_ERR_CUDA, "incidence plan: %s: %s", what, cudaGetErrorString(e));
}

#define PCK(call)                             \
  do {                                        \
    const int rc_ = plan_cuda((call), #call); \
    if (rc_ != LPG_OK) return rc_;            \
  } while (0)

template <typename T>
int dalloc(T** p, size_t n) {
  if (cudaMalloc((void**)p, sizeof(T) * (n ? n : 1)) != cudaSuccess) {
    *p = nullptr;
    return lpg_ops_fail(LPG_ERR_NOMEM, "incidence plan: device allocation of %zu bytes failed", sizeof(T) * n);
  }
  return LPG_OK;
}

void plan_free(lpg_incidence_plan* p) {
  void* ps[] = {p->srisk, p->beta, p->popc, p->doy,  p->year,    p->pops,   p->logp,   p->logd,    p->target,
                p->lp2,   p->ld2,  p->tab,  p->r0s,  p->seas,    p->Gm,     p->rs,     p->rsN,     p->fac,
                p->u,     p->lam,  p->g,    p->gN,   p->sums,    p->N,
                p->small ? p->gu : nullptr, p->b_rows, p->b_cols, p->n_cols, p->gu_cols, p->max_br, p->max_bc,
                p->sq_br, p->sq_bc};
  for (void* q : ps)
    if (q) cudaFree(q);
  if (p->host) cudaFreeHost(p->host);
  for (auto& ev : p->ev)
    if (ev) cudaEventDestroy(ev);
  if (p->own_stream && p->st) cudaStreamDestroy(p->st);
  delete p;
}

/* The shapes of the two sliced products and their depth slices. */
void plan_products(const lpg_incidence_plan* p, OzArgs* mix, OzArgs* flows);

int depth_pad(int k) { return (k + OZ_BK - 1) / OZ_BK * OZ_BK; }

int plan_alloc(lpg_incidence_plan* p) {
  const size_t T = p->T, G = p->G, TG = T * G, TSG = TG * p->S, GG = G * G, TS = T * p->S;
  int rc;
  if ((rc = dalloc(&p->srisk, TG)) || (rc = dalloc(&p->beta, TSG)) || (rc = dalloc(&p->popc, TG)) ||
      (rc = dalloc(&p->doy, T)) || (rc = dalloc(&p->year, T)) || (rc = dalloc(&p->pops, G)) ||
      (rc = dalloc(&p->logp, G)) || (rc = dalloc(&p->logd, GG)) || (rc = dalloc(&p->r0s, G)) ||
      (rc = dalloc(&p->lp2, G)) || (rc = dalloc(&p->ld2, GG)) || (rc = dalloc(&p->tab, 1)) ||
      (rc = dalloc(&p->seas, 3 * T)) || (rc = dalloc(&p->Gm, GG)) || (rc = dalloc(&p->rs, G)) ||
      (rc = dalloc(&p->rsN, G)) || (rc = dalloc(&p->fac, G)) || (rc = dalloc(&p->lam, TG)) ||
      (rc = dalloc(&p->g, TG)) || (rc = dalloc(&p->gN, GG)))
    return rc;
  const size_t clear = SC_N + G + T + 3 * G; /* doubles; the sums of squares two to one */
  if ((rc = dalloc(&p->sums, clear))) return rc;
  p->clear_bytes = clear * sizeof(double);
  p->list_n = reinterpret_cast<unsigned long long*>(p->sums + SC_LIST);
  p->gr0s = p->sums + SC_N;
  p->gw = p->gr0s + G;
  p->max_n = reinterpret_cast<unsigned long long*>(p->gw + T);
  p->max_gu = p->max_n + G;
  p->sq_n = reinterpret_cast<uint32_t*>(p->max_gu + G);
  p->sq_gu = p->sq_n + G;
  if (!p->small) {
    const size_t kg = depth_pad(p->G), kt = depth_pad((int)TS), half = OZ_SLICES / 2; /* two digits a word */
    const size_t tile = OZ_CHUNK * OZ_BK;
    p->row_cap = (int)std::min(TS, TS * kg <= INC_DIGITS ? TS : std::max<size_t>(1, INC_DIGITS / kg / OZ_BM) * OZ_BM);
    p->dep_cap = (int)std::min(kt, kt * G <= INC_DIGITS ? kt : std::max<size_t>(1, INC_DIGITS / G / tile) * tile);
    OzArgs mix{}, flows{};
    plan_products(p, &mix, &flows);
    const size_t words_n = std::max(half * G * kg, 2 * flows.split * GG);
    const size_t words_gu =
        std::max(half * G * p->dep_cap, 2 * std::max(oz_list((int)TS, p->G), oz_list(p->G, p->G)));
    if ((rc = dalloc(&p->u, mix.split * TSG)) || (rc = dalloc(&p->b_rows, half * p->row_cap * kg)) ||
        (rc = dalloc(&p->b_cols, half * G * p->dep_cap)) || (rc = dalloc(&p->n_cols, words_n)) ||
        (rc = dalloc(&p->gu_cols, words_gu)) || (rc = dalloc(&p->max_br, TS)) || (rc = dalloc(&p->max_bc, G)) ||
        (rc = dalloc(&p->sq_br, TS)) || (rc = dalloc(&p->sq_bc, G)))
      return rc;
    p->gu = p->u;
    p->C = reinterpret_cast<double*>(p->n_cols);
    if (!oz_map(&p->map_b, p->b_rows, p->row_cap, (int)kg, OZ_BM) || !oz_map(&p->map_n, p->n_cols, p->G, (int)kg, OZ_BN) ||
        !oz_map(&p->map_bt, p->b_cols, p->G, p->dep_cap, OZ_BM) || !oz_map(&p->map_gu, p->gu_cols, p->G, p->dep_cap, OZ_BN))
      return lpg_ops_fail(LPG_ERR_CUDA, "incidence plan: a tensor map was refused");
  } else if ((rc = dalloc(&p->N, GG)) || (rc = dalloc(&p->gu, TSG))) {
    return rc;
  }
  PCK(cudaMallocHost((void**)&p->host, (SC_N + 2 * G) * sizeof(double)));
  for (auto& ev : p->ev) PCK(cudaEventCreate(&ev));
  return LPG_OK;
}

/* Marks the start of phase ph of an evaluation (and the end of the previous
 * one).  A phase may be several launches, or with the small sums part of
 * another phase's. */
inline void mark(lpg_incidence_plan* p, int ph) {
  if (p->prof) cudaEventRecord(p->ev[ph], p->st);
  p->evals[ph] += 1;
}

void plan_products(const lpg_incidence_plan* p, OzArgs* mix, OzArgs* flows) {
  mix->M = p->row_cap;
  mix->N = p->G;
  mix->k_stages = depth_pad(p->G) / OZ_BK;
  oz_plan(mix, p->nsm, p->row_cap < p->T * p->S ? 1 : INC_MAX_SPLIT); /* parts of u lie side by side: no slabs */
  mix->max_b = p->max_n;
  mix->err = p->sums + SC_ERR;
  mix->polls = flows->polls = p->polls;
  mix->stall = flows->stall = p->stall;
  flows->M = p->G;
  flows->N = p->G;
  flows->k_stages = p->dep_cap / OZ_BK;
  oz_plan(flows, p->nsm, INC_MAX_SPLIT);
  flows->max_a = p->max_bc;
  flows->max_b = p->max_gu;
  flows->C = p->C;
  flows->err = p->sums + SC_ERR;
}

/* The digits of beta's rows [r0, r0 + n), and of depths [k0, k0 + n) by columns. */
void slice_beta_rows(lpg_incidence_plan* p, int r0, int n) {
  const int G = p->G, kg = depth_pad(G);
  k_oz_slice_rows<<<dim3(n, (kg / 2 + 255) / 256), 256, 0, p->st>>>(p->row_cap, G, kg, p->beta + (size_t)r0 * G,
                                                                   p->max_br + r0, p->b_rows, p->sq_br + r0);
}
void slice_beta_cols(lpg_incidence_plan* p, int k0, int n) {
  k_oz_slice_cols<<<dim3((p->G + 31) / 32, depth_pad(n) / 32), 256, 0, p->st>>>(
      n, p->G, p->dep_cap, p->beta + (size_t)k0 * p->G, nullptr, p->max_bc, p->b_cols, p->sq_bc);
}

/* What every evaluation (its gradient) needs of beta beside that: the
 * digits, where a plan keeps them, and the columns' maxima. */
int plan_rows(lpg_incidence_plan* p) {
  const int TS = p->T * p->S;
  if (p->rows_ready) return LPG_OK;
  PCK(cudaMemsetAsync(p->sq_br, 0, sizeof(uint32_t) * TS, p->st));
  if (p->row_cap < TS) return LPG_OK;
  slice_beta_rows(p, 0, TS);
  p->rows_ready = true;
  return plan_cuda(cudaGetLastError(), "slicing");
}
int plan_cols(lpg_incidence_plan* p) {
  const int G = p->G, TS = p->T * p->S;
  if (!p->bc_ready) {
    PCK(cudaMemsetAsync(p->max_bc, 0, sizeof(unsigned long long) * G, p->st));
    k_oz_col_max<<<oz_col_grid(TS, G), 256, 0, p->st>>>(TS, G, p->beta, nullptr, p->max_bc);
    p->bc_ready = true;
  }
  if (p->cols_ready) return LPG_OK;
  PCK(cudaMemsetAsync(p->sq_bc, 0, sizeof(uint32_t) * G, p->st));
  if (p->dep_cap < TS) return LPG_OK;
  slice_beta_cols(p, 0, TS);
  p->cols_ready = true;
  return plan_cuda(cudaGetLastError(), "slicing");
}

/* u = beta N: row_cap rows at a time. */
int plan_mix(lpg_incidence_plan* p, const OzArgs& mix) {
  const int G = p->G, TS = p->T * p->S;
  const int rc = plan_rows(p);
  if (rc != LPG_OK) return rc;
  for (int r0 = 0; r0 < TS; r0 += p->row_cap) {
    OzArgs A = mix;
    A.M = std::min(p->row_cap, TS - r0);
    A.tiles = (A.M + OZ_BM - 1) / OZ_BM * A.tiles_n;
    A.max_a = p->max_br + r0;
    A.C = p->u + (size_t)r0 * G;
    if (!p->rows_ready) slice_beta_rows(p, r0, A.M);
    PCK(oz_gemm(p->map_b, p->map_n, A, p->nsm, p->st));
  }
  PCK(oz_refine<false>(OzRefine{TS, G, G, mix.split, p->beta, p->Gm, p->fac, p->max_br, p->max_n, p->sq_br, p->sq_n,
                                p->u, p->list_n, reinterpret_cast<uint64_t*>(p->gu_cols)},
                       p->nsm, p->st));
  return LPG_OK;
}

/* C = beta^T dL/du: dep_cap depths at a time, added up in C. */
int plan_flows(lpg_incidence_plan* p, const OzArgs& flows) {
  const int G = p->G, TS = p->T * p->S;
  for (int k0 = 0; k0 < TS; k0 += p->dep_cap) {
    const int K = std::min(p->dep_cap, TS - k0), kd = depth_pad(K);
    OzArgs A = flows;
    A.k_stages = kd / OZ_BK;
    A.per_split = (A.k_stages + A.split - 1) / A.split;
    A.add = k0 > 0;
    k_oz_slice_cols<<<dim3((G + 31) / 32, kd / 32), 256, 0, p->st>>>(K, G, p->dep_cap, p->gu + (size_t)k0 * G, nullptr,
                                                                     p->max_gu, p->gu_cols, p->sq_gu);
    if (!p->cols_ready) slice_beta_cols(p, k0, K);
    PCK(oz_gemm(p->map_bt, p->map_gu, A, p->nsm, p->st));
  }
  PCK(oz_refine<true>(OzRefine{G, G, TS, flows.split, p->beta, p->gu, nullptr, p->max_bc, p->max_gu, p->sq_bc, p->sq_gu,
                               p->C, p->list_n + 1, reinterpret_cast<uint64_t*>(p->gu_cols)},
                      p->nsm, p->st));
  return LPG_OK;
}

/* x with 56 fraction bits, |x| < 64. */
int64_t fixed56(double x) { return (int64_t)std::llrint(x * 72057594037927936.0); }

template <bool SMALL>
int launch_step(lpg_incidence_plan* p, const IncStep& A) {
  /* one tick a thread, for latency, until that is 32 CTAs an SM; two beyond,
   * which halves the atomics (774 nodes, 365 ticks: 45 and 47 us; 4000
   * nodes, 90 ticks: 88 and 79 us; eight ticks a thread: 73 and 127) */
  const int gx = (p->G + 127) / 128;
  if ((int64_t)p->T * gx <= 32LL * p->nsm)
    k_inc_step<SMALL, 1><<<dim3(gx, p->T), 128, 0, p->st>>>(p->tab, A);
  else
    k_inc_step<SMALL, 2><<<dim3(gx, (p->T + 1) / 2), 128, 0, p->st>>>(p->tab, A);
  return plan_cuda(cudaGetLastError(), "step launch");
}

int plan_run(lpg_incidence_plan* p, const lpg_incidence_params* prm, IncScalars sc, bool with_loss, const double* g_in,
             bool want_lam, bool grad, bool want_network) {
  const int T = p->T, G = p->G, S = p->S, TS = T * S;
  IncGravity V{prm->a, prm->b, prm->c, prm->k / pow(p->P, prm->c), prm->max_frac, 0, 0, 0, 0};
  auto small = [](double x) { return std::fabs(x) < 60.0; };
  if (small(V.a) && small(V.b) && small(V.c) && std::fabs(V.a) * p->max_lp2 < 900.0 &&
      std::fabs(V.b) * p->max_lp2 + std::fabs(V.c) * p->max_ld2 < 900.0) {
    V.a56 = fixed56(V.a);
    V.b56 = fixed56(V.b);
    V.c56 = fixed56(V.c);
    V.integer = 1;
  }
  OzArgs mix{}, flows{};
  plan_products(p, &mix, &flows);
  mark(p, PH_NETWORK);
  const int nblk = G + (T + 31) / 32;
  if (p->small) {
    k_inc_network<true><<<nblk, INC_THREADS, 0, p->st>>>(G, T, p->tab, p->pops, p->logp, p->logd, p->lp2, p->ld2, V,
                                                         p->Gm, p->N, p->rs, p->rsN, p->fac, p->doy, p->year, sc,
                                                         p->seas);
  } else {
    k_inc_network<false><<<nblk, INC_THREADS, 0, p->st>>>(G, T, p->tab, p->pops, p->logp, p->logd, p->lp2, p->ld2, V,
                                                          p->Gm, nullptr, p->rs, p->rsN, p->fac, p->doy, p->year, sc,
                                                          p->seas);
    k_oz_col_max<<<oz_col_grid(G, G), 256, 0, p->st>>>(G, G, p->Gm, p->fac, p->max_n);
    k_oz_slice_cols<<<dim3((G + 31) / 32, depth_pad(G) / 32), 256, 0, p->st>>>(G, G, depth_pad(G), p->Gm, p->fac,
                                                                              p->max_n, p->n_cols, p->sq_n);
  }
  mark(p, PH_MIX);
  if (!p->small) {
    const int rc = plan_mix(p, mix);
    if (rc != LPG_OK) return rc;
  }
  mark(p, PH_FORWARD);
  IncStep A{};
  A.T = T;
  A.G = G;
  A.S = S;
  A.srisk = p->srisk;
  A.beta = p->beta;
  A.popc = p->popc;
  A.seas = p->seas;
  A.r0s = p->r0s;
  A.rsN = p->rsN;
  A.u = p->u;
  A.N = p->N;
  A.ltarget = with_loss ? p->target : nullptr;
  A.g_in = g_in;
  A.R = sc.R;
  A.lam = want_lam ? p->lam : nullptr;
  A.loss = p->sums + SC_LOSS;
  A.gu = p->gu;
  A.max_gu = p->max_gu;
  A.g_r0s = p->gr0s;
  A.g_w = p->gw;
  A.grad = grad;
  const int rc = p->small ? launch_step<true>(p, A) : launch_step<false>(p, A);
  if (rc != LPG_OK || !grad) return rc;
  mark(p, PH_BACKWARD); /* its cells are part of the step's launch */
  double* gN = want_network ? p->gN : nullptr;
  if (p->small) {
    mark(p, PH_FLOWS);
    mark(p, PH_NETWORK_GRAD);
    const int smem = (int)sizeof(double) * (G > INC_THREADS ? G : INC_THREADS);
    k_inc_network_grad<true><<<G + 1, INC_THREADS, smem, p->st>>>(
        G, T, TS, nullptr, p->beta, p->gu, p->Gm, p->rs, p->fac, p->logp, p->logd, prm->k, p->logP, gN,
        p->sums + SC_THETA, p->seas, p->gw, sc.R, p->sums + SC_R);
  } else {
    int rc = plan_cols(p);
    if (rc != LPG_OK) return rc;
    mark(p, PH_FLOWS);
    rc = plan_flows(p, flows);
    if (rc != LPG_OK) return rc;
    mark(p, PH_NETWORK_GRAD);
    k_inc_network_grad<false><<<(G < 8 * p->nsm ? G : 8 * p->nsm) + 1, INC_THREADS, 0, p->st>>>(
        G, T, TS, p->C, nullptr, nullptr, p->Gm, p->rs, p->fac, p->logp, p->logd, prm->k, p->logP, gN,
        p->sums + SC_THETA, p->seas, p->gw, sc.R, p->sums + SC_R);
  }
  return plan_cuda(cudaGetLastError(), "gradient launch");
}

}  // namespace

extern "C" int lpg_incidence_plan_create(const lpg_incidence_in* in, const double* target, void* stream,
                                         lpg_incidence_plan** out) {
  if (!in || !out) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null argument");
  *out = nullptr;
  const int T = in->T, G = in->G, S = in->S;
  if (T <= 0 || G <= 0 || S <= 0 || S > LPG_MAX_STRAINS)
    return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: bad sizes T=%d G=%d S=%d", T, G, S);
  if ((int64_t)T * S > INC_MAX_ROWS || T > 65535)
    return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: T=%d or T*S = %lld too large (T <= 65535, T*S <= %d)", T,
                        (long long)T * S, INC_MAX_ROWS);
  if (!in->srisk || !in->beta || !in->pop || !in->doy || !in->year || !in->pops || !in->dist)
    return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null input array");
  double P = 0.0;
  for (int i = 0; i < G; ++i) {
    if (!(in->pops[i] >= 0.0)) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: pops[%d] is negative", i);
    P += in->pops[i];
  }
  if (!(P > 0.0) || !std::isfinite(P)) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: total population %g", P);
  /* one pass over the distances: none off the diagonal negative or NaN, and
   * the range of the positive finite ones */
  double dlo = HUGE_VAL, dhi = 0.0;
  for (int i = 0; i < G; ++i) {
    const double* row = in->dist + (size_t)i * G;
    int bad = 0;
    for (int j = 0; j < G; ++j) {
      const double x = row[j];
      bad += !(x >= 0.0);
      const double lo = x > 0.0 ? x : HUGE_VAL, hi = x < HUGE_VAL ? x : 0.0;
      dlo = lo < dlo ? lo : dlo;
      dhi = hi > dhi ? hi : dhi;
    }
    if (bad - !(row[i] >= 0.0))
      for (int j = 0; j < G; ++j)
        if (j != i && !(row[j] >= 0.0))
          return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: dist[%d][%d] is negative", i, j);
  }
  lpg_incidence_plan* p = new lpg_incidence_plan;
  p->T = T;
  p->G = G;
  p->S = S;
  p->P = P;
  p->logP = log(P);
  auto widest = [](double x, double* m) {
    const double l = x > 0.0 && std::isfinite(x) ? std::fabs(std::log2(x)) : 0.0;
    if (l > *m) *m = l;
  };
  for (int i = 0; i < G; ++i) widest(in->pops[i], &p->max_lp2);
  widest(dlo, &p->max_ld2);
  widest(dhi, &p->max_ld2);
  /* the FP64 sums are one chain of G terms a thread; the sliced products take
   * about 80 us with their operands' slicing and refining, whatever their
   * size (an evaluation of 181 ticks, 100 nodes, 2 strains: 100 us in three
   * kernels against 137 in twelve; 244 ticks, 128 nodes: 101 and 143; 21
   * ticks, 333 nodes, 3 strains: 155 and 152) */
  p->small = G <= INC_SMALL_NODES && (int64_t)T * S * G * G <= INC_SMALL_TERMS;
  int rc = LPG_OK;
  int dev = 0;
  rc = plan_cuda(cudaGetDevice(&dev), "device");
  if (rc == LPG_OK) rc = plan_cuda(cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, dev), "SM count");
  if (rc == LPG_OK) {
    if (stream) {
      p->st = (cudaStream_t)stream;
    } else {
      rc = plan_cuda(cudaStreamCreateWithFlags(&p->st, cudaStreamNonBlocking), "stream");
      p->own_stream = rc == LPG_OK;
    }
  }
  if (rc == LPG_OK) rc = plan_alloc(p);
  double* d_dist = nullptr;
  if (rc == LPG_OK) rc = dalloc(&d_dist, (size_t)G * G);
  if (rc == LPG_OK) {
    const size_t TG = (size_t)T * G, GG = (size_t)G * G;
    std::vector<double> bt(TG * S); /* [T][G][S] -> [T][S][G] */
    for (int t = 0; t < T; ++t)
      for (int n = 0; n < G; ++n)
        for (int s = 0; s < S; ++s) bt[((size_t)t * S + s) * G + n] = in->beta[((size_t)t * G + n) * S + s];
    struct {
      double* dst;
      const double* src;
      size_t n;
    } up[] = {{p->srisk, in->srisk, TG},       {p->beta, bt.data(), TG * S},        {p->popc, in->pop, TG},
              {p->doy, in->doy, (size_t)T},    {p->year, in->year, (size_t)T},      {p->pops, in->pops, (size_t)G},
              {d_dist, in->dist, GG}};
    for (auto& c : up) {
      rc = plan_cuda(cudaMemcpyAsync(c.dst, c.src, sizeof(double) * c.n, cudaMemcpyHostToDevice, p->st), "upload");
      if (rc != LPG_OK) break;
    }
    if (rc == LPG_OK && target) {
      rc = dalloc(&p->target, TG);
      if (rc == LPG_OK)
        rc = plan_cuda(cudaMemcpyAsync(p->target, target, sizeof(double) * TG, cudaMemcpyHostToDevice, p->st),
                       "upload target");
    }
    if (rc == LPG_OK)
      rc = plan_cuda(cudaMemcpyAsync(p->tab, ix_tables(), sizeof(IxTables), cudaMemcpyHostToDevice, p->st),
                     "upload tables");
    if (rc == LPG_OK) {
      const size_t cells = GG > TG ? GG : TG;
      k_inc_logs<<<(unsigned)((cells + INC_THREADS - 1) / INC_THREADS), INC_THREADS, 0, p->st>>>(
          p->tab, G, TG, p->pops, d_dist, p->logp, p->logd, p->lp2, p->ld2, p->popc, p->popc, p->target);
      const int TS = T * S;
      if (!p->small) {
        k_oz_row_max<<<(TS + 7) / 8, 256, 0, p->st>>>(TS, G, p->beta, p->max_br);
        rc = plan_rows(p);
        if (rc == LPG_OK && target) rc = plan_cols(p); /* a target is given for its gradient */
      }
      if (rc == LPG_OK) rc = plan_cuda(cudaGetLastError(), "log launch");
    }
    if (rc == LPG_OK) rc = plan_cuda(cudaStreamSynchronize(p->st), "upload sync");
  }
  if (d_dist) cudaFree(d_dist);
  if (rc != LPG_OK) {
    plan_free(p);
    return rc;
  }
  *out = p;
  return LPG_OK;
}

extern "C" int lpg_incidence_plan_eval(lpg_incidence_plan* p, const lpg_incidence_params* prm, const double* g_lam,
                                       double* lam_out, double* loss_out, lpg_incidence_grad* grad) {
  if (!p || !prm || !prm->r0s) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null argument");
  if (grad && !g_lam && !p->target)
    return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: a gradient needs g_lam or a target");
  if (loss_out && !p->target) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: a loss needs a target");
  const int T = p->T, G = p->G;
  const size_t TG = (size_t)T * G, GG = (size_t)G * G;
  const IncScalars sc{prm->R, prm->amp, prm->peak};
  const bool with_loss = p->target != nullptr && (!g_lam || loss_out);
  double* h_r0s = p->host + SC_N + G;
  for (int i = 0; i < G; ++i) h_r0s[i] = prm->r0s[i];
  PCK(cudaMemcpyAsync(p->r0s, h_r0s, sizeof(double) * G, cudaMemcpyHostToDevice, p->st));
  PCK(cudaMemsetAsync(p->sums, 0, p->clear_bytes, p->st));
  if (grad && g_lam) PCK(cudaMemcpyAsync(p->g, g_lam, sizeof(double) * TG, cudaMemcpyHostToDevice, p->st));
  const bool want_network = grad && grad->network;
  const int rc = plan_run(p, prm, sc, with_loss, grad && g_lam ? p->g : nullptr, lam_out != nullptr, grad != nullptr,
                          want_network);
  if (rc != LPG_OK) return rc;
  if (p->prof) PCK(cudaEventRecord(p->ev[PH_COUNT], p->st));
  PCK(cudaMemcpyAsync(p->host, p->sums, sizeof(double) * (SC_N + (grad ? G : 0)), cudaMemcpyDeviceToHost, p->st));
  if (lam_out) PCK(cudaMemcpyAsync(lam_out, p->lam, sizeof(double) * TG, cudaMemcpyDeviceToHost, p->st));
  if (want_network) PCK(cudaMemcpyAsync(grad->network, p->gN, sizeof(double) * GG, cudaMemcpyDeviceToHost, p->st));
  PCK(cudaStreamSynchronize(p->st));
  if (p->host[SC_ERR] != 0.0) return lpg_ops_fail(LPG_ERR_TIMEOUT, "incidence plan: a product's wait ran out");
  if (p->prof) {
    const int last = grad ? PH_COUNT : PH_BACKWARD;
    for (int ph = 0; ph < last; ++ph) {
      float ms = 0.f;
      const int nxt = ph + 1 == last ? PH_COUNT : ph + 1;
      PCK(cudaEventElapsedTime(&ms, p->ev[ph], p->ev[nxt]));
      p->ms[ph] += ms;
    }
  }
  if (loss_out) *loss_out = p->host[SC_LOSS];
  if (grad) {
    if (grad->r0s)
      for (int i = 0; i < G; ++i) grad->r0s[i] = p->host[SC_N + i];
    grad->R = p->host[SC_R];
    grad->amp = p->host[SC_R + 1];
    grad->peak = p->host[SC_R + 2];
    grad->k = p->host[SC_THETA];
    grad->a = p->host[SC_THETA + 1];
    grad->b = p->host[SC_THETA + 2];
    grad->c = p->host[SC_THETA + 3];
  }
  return LPG_OK;
}

extern "C" void* lpg_incidence_plan_stream(lpg_incidence_plan* p) { return p ? (void*)p->st : nullptr; }

extern "C" int lpg_test_stall_products(lpg_incidence_plan* p, int32_t stages, int64_t wait_polls) {
  if (!p) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null argument");
  if (wait_polls < 0 || wait_polls > OZ_WAIT_POLLS)
    return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: wait_polls %lld out of range", (long long)wait_polls);
  p->stall = stages < 0 ? -1 : stages;
  p->polls = wait_polls > 0 ? (int)wait_polls : OZ_WAIT_POLLS;
  return LPG_OK;
}

extern "C" int lpg_incidence_plan_set_profiling(lpg_incidence_plan* p, int32_t enable) {
  if (!p) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null argument");
  p->prof = enable != 0;
  for (int ph = 0; ph < PH_COUNT; ++ph) {
    p->ms[ph] = 0.0;
    p->evals[ph] = 0;
  }
  return LPG_OK;
}

extern "C" int lpg_incidence_plan_read_profile(lpg_incidence_plan* p, lpg_profile* out) {
  if (!p || !out) return lpg_ops_fail(LPG_ERR_ARG, "incidence plan: null argument");
  *out = lpg_profile{};
  out->n_kernels = PH_COUNT;
  for (int ph = 0; ph < PH_COUNT; ++ph) {
    out->names[ph] = kPhaseNames[ph];
    out->total_ms[ph] = p->ms[ph];
    out->launches[ph] = p->evals[ph];
  }
  return LPG_OK;
}

extern "C" void lpg_incidence_plan_destroy(lpg_incidence_plan* p) {
  if (p) plan_free(p);
}

extern "C" int lpg_expected_incidence(const lpg_incidence_in* in, double* lam_out, const double* g_lam,
                                      lpg_incidence_grad* grad, void* stream) {
  if (!in || !lam_out) return lpg_ops_fail(LPG_ERR_ARG, "expected_incidence: null argument");
  if (g_lam && !grad) return lpg_ops_fail(LPG_ERR_ARG, "expected_incidence: a gradient needs grad");
  if (!in->r0s) return lpg_ops_fail(LPG_ERR_ARG, "expected_incidence: null input array");
  lpg_incidence_plan* p = nullptr;
  int rc = lpg_incidence_plan_create(in, nullptr, stream, &p);
  if (rc != LPG_OK) return rc;
  const lpg_incidence_params prm{in->R, in->amp, in->peak, in->k, in->a, in->b, in->c, in->max_frac, in->r0s};
  rc = lpg_incidence_plan_eval(p, &prm, g_lam, lam_out, nullptr, g_lam ? grad : nullptr);
  lpg_incidence_plan_destroy(p);
  return rc;
}
