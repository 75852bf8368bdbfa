/*
 * lpg_ops.cu — standalone per-node state counts over plain device columns.
 *
 * lpg_count_seirp restates count_SEIRP (laser_polio/model.py:869-899) and
 * its kernel (:902-929): for every slot with disease_state >= 0, count it
 * into S / E_by_strain / I_by_strain / R of its node by state, and into
 * potentially_paralyzed / paralyzed when those flags equal 1; E and I are
 * the per-node sums over strains.  The reference reduces numba thread-local
 * tables; here every CTA builds a node x field histogram in shared memory
 * and adds its entries that are not zero to the outputs, which a small
 * kernel clears first (a count that fits one CTA is stored directly, in one
 * launch).  Integer counts, so the result is exact and does not depend on
 * the order.  No scratch and no allocation.
 *
 * lpg_count_seirp and lpg_count_seirp_static are the same operation; the
 * second keeps the name it had when the first allocated its scratch.
 */
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <mutex>

#include "lpg.h"

#define SEIRP_THREADS 512
#define SEIRP_APT 16        /* slots per thread and step */
#define SEIRP_TILE_STEPS 8  /* steps a warp takes before it adds up: 252 us; 16: 280, 4: 261 (2.2e8 slots) */
#define SEIRP_ONE_CTA (4 * SEIRP_THREADS * SEIRP_APT) /* slots: one CTA, one launch up to here */
#define SEIRP_FIELDS_MAX (4 + 2 * LPG_MAX_STRAINS)
#define SEIRP_MAX_DEVICES 64

/* Field layout of one histogram: [field][node], then one word holding the
 * number of invalid slots.  Fields: 0 S, 1 R, 2 potentially_paralyzed,
 * 3 paralyzed, 4.. E by strain, 4+ns.. I by strain. */
struct SeirpIn {
  const int16_t* node;
  const int8_t* ds;
  const int8_t* strain;
  const int8_t* pp;
  const int8_t* par;
  int64_t n;
  int32_t G, ns, F, tile_steps;
};

struct SeirpOut {
  int32_t *S, *E, *I, *R, *Ebs, *Ibs, *POTP, *P;
  int64_t* n_invalid;
};

static thread_local char g_err[256] = "";

static int op_fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

/* The same error text for the ops of other translation units (lpg_adjoint.cu). */
int lpg_ops_fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}

extern "C" const char* lpg_op_last_error(void) { return g_err; }

/* ------------------------------------------------------------------------ */
/* count_SEIRP_kernel's body for one slot (model.py:913-929).  Slots whose
 * node id lies outside [0, G), or which are E/I with a strain outside
 * [0, ns), are counted as invalid instead (the reference indexes out of
 * bounds there). */
__device__ __forceinline__ void seirp_slot(int32_t* h, const SeirpIn& a, int8_t s, int nd, int8_t st, int8_t pp,
                                           int8_t pa, int32_t& bad) {
  /* without branches but the atomics': neighbouring slots take different ones */
  const bool live = s >= 0, in = (unsigned)nd < (unsigned)a.G, ei = s == 1 || s == 2, known = (unsigned)st < (unsigned)a.ns;
  const int f = s == 0 ? 0 : s == 3 ? 1 : 4 + (s - 1) * a.ns + st;
  const bool counted = live && in;
  bad += live && (!in || (ei && !known));
  if (counted && s <= 3 && (!ei || known)) atomicAdd(&h[f * a.G + nd], 1);
  if (counted && pp == 1) atomicAdd(&h[2 * a.G + nd], 1);
  if (counted && pa == 1) atomicAdd(&h[3 * a.G + nd], 1);
}

__device__ __forceinline__ uint32_t word_of(const uint4& v, int j) {
  return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
}

/* 0x80 in every byte of w that equals k. */
__device__ __forceinline__ uint32_t bytes_equal(uint32_t w, uint32_t k) {
  const uint32_t x = w ^ (k * 0x01010101u);
  return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;
}

/* A thread's counts of one node: four byte lanes a field, at most four more
 * each a step, so that a tile's steps stay below 256. */
struct SeirpAcc {
  uint32_t f[4], e[LPG_MAX_STRAINS], i[LPG_MAX_STRAINS];
};
static_assert(4 * SEIRP_TILE_STEPS < 256, "byte counters");

__device__ __forceinline__ void seirp_clear(SeirpAcc& c) {
#pragma unroll
  for (int k = 0; k < 4; ++k) c.f[k] = c.e[k] = c.i[k] = 0;
}

__device__ __forceinline__ uint32_t byte_sum(uint32_t v) { return __dp4a(v, 0x01010101u, 0u); }

/* One thread's counts of node cur into the histogram. */
__device__ __forceinline__ void seirp_flush(int32_t* h, const SeirpIn& a, int cur, SeirpAcc& c) {
  if (cur < 0) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (c.f[k]) atomicAdd(&h[k * a.G + cur], (int32_t)byte_sum(c.f[k]));
    if (c.e[k]) atomicAdd(&h[(4 + k) * a.G + cur], (int32_t)byte_sum(c.e[k]));
    if (c.i[k]) atomicAdd(&h[(4 + a.ns + k) * a.G + cur], (int32_t)byte_sum(c.i[k]));
  }
  seirp_clear(c);
}

/* One CTA: histogram of its slots in shared memory, then its entries that
 * are not zero added to the outputs (DIRECT: the only CTA, all stored).
 * VEC: warps take tiles of consecutive slots, 16 a lane and step with 16-byte
 * loads (every column 16-byte aligned).  Sixteen slots of one node, nearly
 * all of a table in node order, are counted four bytes an operation and added
 * up once a tile and warp; others slot by slot, as is the tail past the last
 * full group and the whole range when VEC is false.  Bound by HBM: 2.2e8 slots of
 * 774 nodes in 252 us (6 bytes a slot); one run-length state machine a
 * slot took 800. */
template <bool VEC, bool DIRECT>
__global__ void __launch_bounds__(SEIRP_THREADS, 2) k_seirp(SeirpIn a, SeirpOut o) {
  extern __shared__ int32_t h[];
  __shared__ int s_next;
  const int slice = a.F * a.G + 1;
  if (threadIdx.x == 0) s_next = 0;
  for (int i = threadIdx.x; i < slice; i += blockDim.x) h[i] = 0;
  __syncthreads();
  int32_t bad = 0;
  int64_t tail0 = 0;
  if (VEC) {
    const int lane = threadIdx.x & 31;
    const int64_t groups = a.n / SEIRP_APT;
    tail0 = groups * SEIRP_APT;
    const int64_t tile = (int64_t)a.tile_steps * 32, tiles = (groups + tile - 1) / tile;
    for (;;) {
      /* the CTA's next tile: tiles of mixed nodes take a warp several times as long */
      int q = 0;
      if (lane == 0) q = atomicAdd(&s_next, 1);
      const int64_t t = blockIdx.x + (int64_t)__shfl_sync(0xffffffffu, q, 0) * gridDim.x;
      if (t >= tiles) break;
      SeirpAcc c;
      seirp_clear(c);
      int cur = -1;
      const int64_t g1 = min(groups, (t + 1) * tile);
#pragma unroll 2
      for (int64_t g = t * tile + lane; g < g1; g += 32) {
        const int64_t i0 = g * SEIRP_APT;
        const uint4 vds = __ldg(reinterpret_cast<const uint4*>(a.ds + i0));
        const uint4 vst = __ldg(reinterpret_cast<const uint4*>(a.strain + i0));
        const uint4 vpp = __ldg(reinterpret_cast<const uint4*>(a.pp + i0));
        const uint4 vpa = __ldg(reinterpret_cast<const uint4*>(a.par + i0));
        const uint4 n0 = __ldg(reinterpret_cast<const uint4*>(a.node + i0));
        const uint4 n1 = __ldg(reinterpret_cast<const uint4*>(a.node + i0 + 8));
        const uint32_t nd = n0.x & 0xffffu, two = nd * 0x10001u;
        if ((((n0.x ^ two) | (n0.y ^ two) | (n0.z ^ two) | (n0.w ^ two) | (n1.x ^ two) | (n1.y ^ two) | (n1.z ^ two) |
              (n1.w ^ two)) == 0) && nd < (uint32_t)a.G) {
          if ((int)nd != cur) {
            seirp_flush(h, a, cur, c);
            cur = (int)nd;
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t ds = word_of(vds, j), st = word_of(vst, j);
            const uint32_t live = ~ds & 0x80808080u;
            const uint32_t mE = bytes_equal(ds, 1), mI = bytes_equal(ds, 2);
            c.f[0] += bytes_equal(ds, 0) >> 7;
            c.f[1] += bytes_equal(ds, 3) >> 7;
            c.f[2] += (bytes_equal(word_of(vpp, j), 1) & live) >> 7;
            c.f[3] += (bytes_equal(word_of(vpa, j), 1) & live) >> 7;
            if (mE | mI) {
              uint32_t other = mE | mI;
#pragma unroll
              for (int k = 0; k < LPG_MAX_STRAINS; ++k) {
                if (k >= a.ns) break;
                const uint32_t m = bytes_equal(st, (uint32_t)k);
                c.e[k] += (mE & m) >> 7;
                c.i[k] += (mI & m) >> 7;
                other &= ~m;
              }
              bad += __popc(other);
            }
          }
        } else {
#pragma unroll 4
          for (int j = 0; j < SEIRP_APT; ++j) {
            const int b = 8 * (j & 3);
            const uint32_t nw = j < 8 ? word_of(n0, j >> 1) : word_of(n1, (j >> 1) - 4);
            seirp_slot(h, a, (int8_t)(word_of(vds, j >> 2) >> b), (int)(int16_t)(nw >> 16 * (j & 1)),
                       (int8_t)(word_of(vst, j >> 2) >> b), (int8_t)(word_of(vpp, j >> 2) >> b),
                       (int8_t)(word_of(vpa, j >> 2) >> b), bad);
          }
        }
      }
      /* the warp's lanes mostly hold one node: one sum and one atomic a field */
      const int lead = __shfl_sync(0xffffffffu, cur, 0);
      if (__all_sync(0xffffffffu, cur == lead)) {
        if (lead >= 0) {
#pragma unroll
          for (int f = 0; f < SEIRP_FIELDS_MAX; ++f) {
            const uint32_t v = f < 4 ? c.f[f] : f < 4 + LPG_MAX_STRAINS ? c.e[f - 4] : c.i[f - 4 - LPG_MAX_STRAINS];
            const int32_t sum = (int32_t)__reduce_add_sync(0xffffffffu, byte_sum(v));
            const int at = f < 4 + LPG_MAX_STRAINS ? f : f - LPG_MAX_STRAINS + a.ns;
            if (lane == 0 && sum) atomicAdd(&h[at * a.G + lead], sum);
          }
        }
      } else {
        seirp_flush(h, a, cur, c);
      }
    }
  }
  for (int64_t i = tail0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x)
    seirp_slot(h, a, a.ds[i], a.node[i], a.strain[i], a.pp[i], a.par[i], bad);
  if (bad) atomicAdd(&h[slice - 1], bad);
  __syncthreads();
  if (DIRECT) {
    for (int nd = threadIdx.x; nd < a.G; nd += blockDim.x) {
      o.S[nd] = h[nd];
      o.R[nd] = h[a.G + nd];
      o.POTP[nd] = h[2 * a.G + nd];
      o.P[nd] = h[3 * a.G + nd];
      int32_t e = 0, i = 0;
      for (int k = 0; k < a.ns; ++k) {
        const int32_t ek = h[(4 + k) * a.G + nd], ik = h[(4 + a.ns + k) * a.G + nd];
        o.Ebs[(int64_t)nd * a.ns + k] = ek;
        o.Ibs[(int64_t)nd * a.ns + k] = ik;
        e += ek;
        i += ik;
      }
      o.E[nd] = e;
      o.I[nd] = i;
    }
    if (threadIdx.x == 0 && o.n_invalid) *o.n_invalid = h[slice - 1];
  } else {
    for (int at = threadIdx.x; at < slice - 1; at += blockDim.x) {
      const int32_t v = h[at];
      if (!v) continue;
      const int f = at / a.G, nd = at - f * a.G;
      if (f < 4) {
        atomicAdd(&(f == 0 ? o.S : f == 1 ? o.R : f == 2 ? o.POTP : o.P)[nd], v);
      } else if (f < 4 + a.ns) {
        atomicAdd(&o.Ebs[(int64_t)nd * a.ns + f - 4], v);
        atomicAdd(&o.E[nd], v);
      } else {
        atomicAdd(&o.Ibs[(int64_t)nd * a.ns + f - 4 - a.ns], v);
        atomicAdd(&o.I[nd], v);
      }
    }
    if (threadIdx.x == 0 && o.n_invalid && h[slice - 1])
      atomicAdd(reinterpret_cast<unsigned long long*>(o.n_invalid), (unsigned long long)h[slice - 1]);
  }
}

__global__ void __launch_bounds__(256) k_seirp_clear(SeirpOut o, int32_t G, int32_t ns) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < G * ns) o.Ebs[i] = o.Ibs[i] = 0;
  if (i < G) o.S[i] = o.E[i] = o.I[i] = o.R[i] = o.POTP[i] = o.P[i] = 0;
  if (i == 0 && o.n_invalid) *o.n_invalid = 0;
}

/* ------------------------------------------------------------------------ */
/* Per-device setup: SM count, and the kernels' dynamic shared memory opt-in
 * (up to SEIRP_FIELDS_MAX x LPG_COUNT_SEIRP_MAX_NODES + 1 words). */
struct SeirpDev {
  bool ready;
  int sms;
};
static SeirpDev g_dev[SEIRP_MAX_DEVICES];
static std::mutex g_dev_mu;

static const size_t kSmemMax = ((size_t)SEIRP_FIELDS_MAX * LPG_COUNT_SEIRP_MAX_NODES + 1) * sizeof(int32_t);

static int seirp_dev_setup(int dev, int* sms) {
  std::lock_guard<std::mutex> lk(g_dev_mu);
  SeirpDev& d = g_dev[dev];
  if (!d.ready) {
    cudaError_t e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    void (*const ks[])(SeirpIn, SeirpOut) = {k_seirp<true, true>, k_seirp<true, false>, k_seirp<false, true>,
                                             k_seirp<false, false>};
    for (auto k : ks)
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
    if (e != cudaSuccess) return op_fail(LPG_ERR_CUDA, "count_SEIRP setup: %s", cudaGetErrorString(e));
    d.ready = true;
  }
  *sms = d.sms;
  return LPG_OK;
}

extern "C" int lpg_count_seirp(const int16_t* node_id, const int8_t* disease_state, const int8_t* strain,
                               const int8_t* potentially_paralyzed, const int8_t* paralyzed, int32_t n_nodes,
                               int32_t n_strains, int64_t n_people, int32_t* S, int32_t* E, int32_t* I, int32_t* R,
                               int32_t* E_by_strain, int32_t* I_by_strain, int32_t* POTP, int32_t* P,
                               int64_t* n_invalid, void* stream) {
  if (n_nodes < 1 || n_nodes > LPG_COUNT_SEIRP_MAX_NODES)
    return op_fail(LPG_ERR_ARG, "count_SEIRP: n_nodes %d outside [1, %d]", n_nodes, LPG_COUNT_SEIRP_MAX_NODES);
  if (n_strains < 1 || n_strains > LPG_MAX_STRAINS)
    return op_fail(LPG_ERR_ARG, "count_SEIRP: n_strains %d outside [1, %d]", n_strains, LPG_MAX_STRAINS);
  if (n_people < 0) return op_fail(LPG_ERR_ARG, "count_SEIRP: n_people %lld < 0", (long long)n_people);
  if (n_people > 0 && (!node_id || !disease_state || !strain || !potentially_paralyzed || !paralyzed))
    return op_fail(LPG_ERR_ARG, "count_SEIRP: a column pointer is NULL");
  if (!S || !E || !I || !R || !E_by_strain || !I_by_strain || !POTP || !P)
    return op_fail(LPG_ERR_ARG, "count_SEIRP: an output pointer is NULL");
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return op_fail(LPG_ERR_CUDA, "count_SEIRP: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= SEIRP_MAX_DEVICES) return op_fail(LPG_ERR_ARG, "count_SEIRP: device %d", dev);
  const int rc = seirp_dev_setup(dev, &sms);
  if (rc) return rc;
  auto al16 = [](const void* p) { return ((uintptr_t)p & 15u) == 0; };
  const bool vec = al16(node_id) && al16(disease_state) && al16(strain) && al16(potentially_paralyzed) && al16(paralyzed);
  SeirpIn in{node_id, disease_state, strain, potentially_paralyzed, paralyzed, n_people,
             n_nodes, n_strains, 4 + 2 * n_strains, 1};
  const SeirpOut out{S, E, I, R, E_by_strain, I_by_strain, POTP, P, n_invalid};
  const size_t smem = ((size_t)in.F * n_nodes + 1) * sizeof(int32_t);
  const cudaStream_t st = (cudaStream_t)stream;
  if (n_people <= SEIRP_ONE_CTA) {
    if (vec) k_seirp<true, true><<<1, SEIRP_THREADS, smem, st>>>(in, out);
    else k_seirp<false, true><<<1, SEIRP_THREADS, smem, st>>>(in, out);
  } else {
    /* two CTAs an SM while their histograms fit; tiles of up to
     * SEIRP_TILE_STEPS steps, shorter when every warp then still has one */
    const int per_sm = 2 * (smem + 1024) <= 227 * 1024 ? 2 : 1;
    const int64_t step = (int64_t)SEIRP_THREADS * SEIRP_APT;
    const int nblk = (int)std::min<int64_t>((n_people + step - 1) / step, (int64_t)per_sm * sms);
    in.tile_steps = (int32_t)std::min<int64_t>(SEIRP_TILE_STEPS, (n_people + step * nblk - 1) / (step * nblk));
    k_seirp_clear<<<(n_nodes * n_strains + 255) / 256, 256, 0, st>>>(out, n_nodes, n_strains);
    if (vec) k_seirp<true, false><<<nblk, SEIRP_THREADS, smem, st>>>(in, out);
    else k_seirp<false, false><<<nblk, SEIRP_THREADS, smem, st>>>(in, out);
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return op_fail(LPG_ERR_CUDA, "count_SEIRP launch: %s", cudaGetErrorString(e));
  return LPG_OK;
}

extern "C" int lpg_count_seirp_static(const int16_t* node_id, const int8_t* disease_state, const int8_t* strain,
                                      const int8_t* potentially_paralyzed, const int8_t* paralyzed, int32_t n_nodes,
                                      int32_t n_strains, int64_t n_people, int32_t* S, int32_t* E, int32_t* I,
                                      int32_t* R, int32_t* E_by_strain, int32_t* I_by_strain, int32_t* POTP,
                                      int32_t* P, int64_t* n_invalid, void* stream) {
  return lpg_count_seirp(node_id, disease_state, strain, potentially_paralyzed, paralyzed, n_nodes, n_strains, n_people,
                         S, E, I, R, E_by_strain, I_by_strain, POTP, P, n_invalid, stream);
}
