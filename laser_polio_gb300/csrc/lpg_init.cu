/*
 * lpg_init.cu — the model's initialisation on the device (lpg_init_columns).
 *
 * The reference builds its agent table on the host with numpy
 * (model.py:101-175, 561-713, 816-866, 1548-1611, 1887-1894), minutes at
 * Nigeria scale.  Here:
 *   - the per-slot columns are filled in grid-stride passes over the capacity
 *     (lpg_init.h holds the arithmetic, shared with the oracle): constants and
 *     node ids by k_init_base, dates by k_init_dates, timers and heterogeneity
 *     by lpg_init_fast.cuh's kernels, or by k_init_slots in FP64 where the
 *     parameters have no fast form;
 *   - the choices without replacement (chronically missed, immune and
 *     initially infected agents) take, in each group, the k agents with the
 *     smallest counter-based 64-bit keys, ties by slot.  Keys are uniform, so
 *     the k-th smallest of n lies within a few sqrt(k (n - k) / n) / n of k / n:
 *     one pass over the agents forms each key once, keeps a bit for the keys
 *     below that window, counts them, and lists the few inside it; a CTA per
 *     group picks the missing ones from its list; a last pass over the bits
 *     marks.  Were the window to miss (it is 7 standard deviations either
 *     side), the choice is made again with a wider one.  Scratch: a bit an
 *     agent and 16 bytes a listed key.
 * Groups are whole nodes (the initial table is node-contiguous) or the whole
 * population.  Everything is HBM-light integer work: the passes are bound by
 * Philox arithmetic (about 140 integer instructions per key).  The timers
 * and the heterogeneity, whose definitions are FP64, have FP32 forms with
 * the same bits (lpg_init_fast.cuh).
 */
#include <cuda_runtime.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <vector>

#include "lpg.h"
#include "lpg_init.h"
#include "lpg_init_fast.cuh"

int lpg_ops_fail(int code, const char* fmt, ...);

namespace {

constexpr int kTile = 8192; /* slots per CTA tile of the selection's pass */
constexpr int kThreads = 256;

struct SlotArgs {
  uint64_t seed;
  int64_t count, capacity;
  int32_t n_nodes, n_bins;
  const int64_t* node_start; /* [n_nodes + 1] */
  int32_t k_exp, k_inf, k_par, het;
  double e1, e2, i1, i2, p1, p2;
  double mu, sigma, rho, srho, scale;
  const int64_t* age_cum;
  const int32_t* age_lo;
  const int32_t* age_hi;
  const int64_t* km;
  int32_t km_len, km_max_year;
};

__device__ __forceinline__ int32_t group_of(const int64_t* start, int32_t n, int64_t slot) {
  int32_t a = 0, b = n - 1; /* last group with start <= slot */
  while (a < b) {
    const int32_t m = (a + b + 1) >> 1;
    if (start[m] <= slot) a = m; else b = m - 1;
  }
  return a;
}

/* The parts that fill constants and node ids, 16 slots a thread and step:
 * one node search and 16-byte stores where the columns allow them. */
__device__ __forceinline__ void fill_base(const SlotArgs& A, const lpg_columns& c, int64_t i0, bool wide) {
  if (wide && i0 + 16 <= A.capacity && (i0 + 16 <= A.count || i0 >= A.count)) {
    const bool live = i0 < A.count;
    const uint4 zero = make_uint4(0, 0, 0, 0), ones = make_uint4(~0u, ~0u, ~0u, ~0u);
    *reinterpret_cast<uint4*>(c.disease_state + i0) = live ? zero : ones;
    *reinterpret_cast<uint4*>(c.strain + i0) = zero;
    *reinterpret_cast<uint4*>(c.potentially_paralyzed + i0) = ones;
    *reinterpret_cast<uint4*>(c.paralyzed + i0) = zero;
    *reinterpret_cast<uint4*>(c.ipv_protected + i0) = zero;
    *reinterpret_cast<uint4*>(c.chronically_missed + i0) = zero;
    uint32_t w[8];
    if (!live) {
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = ~0u;
    } else {
      int32_t g = group_of(A.node_start, A.n_nodes, i0);
      if (A.node_start[g + 1] >= i0 + 16) {
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = (uint32_t)g * 0x10001u;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t lo = (uint32_t)group_of(A.node_start, A.n_nodes, i0 + 2 * j);
          w[j] = lo | (uint32_t)group_of(A.node_start, A.n_nodes, i0 + 2 * j + 1) << 16;
        }
      }
    }
    uint4* d = reinterpret_cast<uint4*>(c.node_id + i0);
    d[0] = make_uint4(w[0], w[1], w[2], w[3]);
    d[1] = make_uint4(w[4], w[5], w[6], w[7]);
    return;
  }
  for (int64_t i = i0; i < i0 + 16 && i < A.capacity; ++i) {
    const bool live = i < A.count;
    c.disease_state[i] = live ? 0 : -1;
    c.node_id[i] = live ? (int16_t)group_of(A.node_start, A.n_nodes, i) : (int16_t)-1;
    c.strain[i] = 0;
    c.potentially_paralyzed[i] = -1;
    c.paralyzed[i] = 0;
    c.ipv_protected[i] = 0;
    c.chronically_missed[i] = 0;
  }
}

__global__ void __launch_bounds__(kThreads) k_init_base(SlotArgs A, lpg_columns c, bool wide) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x * 16;
  for (int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 16; i0 < A.capacity; i0 += stride)
    fill_base(A, c, i0, wide);
}

__global__ void __launch_bounds__(kThreads) k_init_slots(SlotArgs A, lpg_columns c, uint32_t parts) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.capacity; i += stride) {
    if (parts & LPG_INIT_TIMERS)
      lpg_init_timers(A.seed, (uint64_t)i, A.k_exp, A.e1, A.e2, A.k_inf, A.i1, A.i2, A.k_par, A.p1, A.p2,
                      &c.exposure_timer[i], &c.infection_timer[i], &c.paralysis_timer[i]);
    if (parts & LPG_INIT_HETEROGENEITY)
      lpg_init_het(A.seed, (uint64_t)i, A.het, A.mu, A.sigma, A.rho, A.srho, A.scale, &c.acq_risk_multiplier[i],
                   &c.daily_infectivity[i]);
  }
}

/* Dates of birth and death and RI dates.  Bound by Philox (a block each);
 * with searches of seven steps in global memory and FP64 scaling 2.3e8 slots
 * took 11.3 ms. */
__global__ void __launch_bounds__(kThreads) k_init_dates(SlotArgs A, lpg_columns c, uint32_t parts) {
  __shared__ FiDates D;
  fi_dates_load(D, parts & LPG_INIT_AGES ? A.age_cum : nullptr, A.age_lo, A.age_hi, A.n_bins,
                parts & LPG_INIT_DEATHS ? A.km : nullptr, A.km_len, A.km_max_year);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < A.capacity; i += stride) {
    const bool live = i < A.count;
    int32_t dob = -1;
    if (parts & LPG_INIT_AGES) {
      dob = live ? -fi_age(D, A.seed, (uint64_t)i) : -1;
      c.date_of_birth[i] = dob;
    } else {
      dob = c.date_of_birth[i];
    }
    if (parts & LPG_INIT_DEATHS) {
      int32_t dod = 0;
      if (live) {
        const int64_t age = -(int64_t)dob;
        uint64_t w[4] = {(uint64_t)i, 0, (uint64_t)LPG_P_INIT_KM << 32, 0};
        lpg_philox4x64_10(w, A.seed, LPG_KEY_TAG);
        dod = (int32_t)(fi_age_at_death(D, age, w[0] >> 11, w[1] >> 11) - age);
      }
      c.date_of_death[i] = dod;
    }
    if (parts & LPG_INIT_RI) c.ri_timer[i] = live ? fi_ri(A.seed, (uint64_t)i, dob) : (int16_t)-1;
  }
}

/* --- selection of k agents per group by their smallest keys ------------- */
struct SelGroup {
  int64_t start;     /* first agent; the next group's start ends it */
  int64_t k;         /* <= 0: none, >= size: all */
  uint64_t lo, hi;   /* keys below lo are taken, keys in [lo, hi] listed */
  int64_t list, cap; /* the group's part of the list */
};
struct SelKey {
  uint64_t key;
  int64_t slot;
};
struct Sel {
  uint64_t seed;
  uint32_t purpose;
  int32_t n_groups;
  const SelGroup* g;          /* [n_groups + 1] */
  unsigned long long* below;  /* [n_groups] */
  unsigned long long* listed; /* [n_groups] */
  SelKey* list;
  uint32_t* bits; /* one per agent */
  int* err;       /* a window that missed */
};

__device__ __forceinline__ int32_t sel_group(const Sel& S, int64_t slot) {
  int32_t a = 0, b = S.n_groups - 1;
  while (a < b) {
    const int32_t m = (a + b + 1) >> 1;
    if (S.g[m].start <= slot) a = m; else b = m - 1;
  }
  return a;
}

/* Bound by Philox (the 64-bit products: 2.1 ms for 2.2e8 blocks).  2.2e8
 * agents in 774 nodes chosen and marked in 3.3 ms; four passes for the keys'
 * digits and a marking one, a Philox block an agent each, took 14.6. */
__global__ void __launch_bounds__(kThreads) k_rsel_pass(Sel S, int64_t count) {
  const int lane = threadIdx.x & 31;
  for (int64_t t0 = (int64_t)blockIdx.x * kTile; t0 < count; t0 += (int64_t)gridDim.x * kTile) {
    const int64_t t1 = t0 + kTile < count ? t0 + kTile : count;
    const int32_t g0 = sel_group(S, t0);
    const bool one = S.g[g0 + 1].start >= t1; /* the tile lies in one group */
    const SelGroup G0 = S.g[g0];
    const int64_t n0 = S.g[g0 + 1].start - G0.start;
    uint32_t below = 0;
    for (int64_t i0 = t0 + (threadIdx.x & ~31); i0 < t1; i0 += blockDim.x) {
      const int64_t i = i0 + lane;
      bool take = false, inside = false;
      int32_t g = g0;
      uint64_t key = 0;
      if (i < t1) {
        if (!one) g = sel_group(S, i);
        const int64_t k = one ? G0.k : S.g[g].k, n = one ? n0 : S.g[g + 1].start - S.g[g].start;
        if (k >= n) {
          take = true;
        } else if (k > 0) {
          key = lpg_raw(S.seed, S.purpose, 0, (uint64_t)i, 0, 0);
          const uint64_t lo = one ? G0.lo : S.g[g].lo, hi = one ? G0.hi : S.g[g].hi;
          take = key < lo;
          inside = !take && key <= hi;
          if (take && !one) atomicAdd(&S.below[g], 1ULL);
        }
      }
      const uint32_t word = __ballot_sync(0xffffffffu, take);
      if (lane == 0) {
        S.bits[i0 >> 5] = word; /* tiles start at multiples of 32 */
        below += __popc(word);
      }
      if (inside) {
        const unsigned long long at = atomicAdd(&S.listed[g], 1ULL);
        const SelGroup& G = S.g[g];
        if ((int64_t)at < G.cap) S.list[G.list + at] = SelKey{key, i};
      }
    }
    if (one && lane == 0 && below && G0.k < n0) atomicAdd(&S.below[g0], (unsigned long long)below);
  }
}

__device__ __forceinline__ void sel_apply(const lpg_columns& c, int action, int64_t i) {
  if (action == 0) c.chronically_missed[i] = 1;
  else if (action == 1) c.disease_state[i] = 3;
  else c.disease_state[i] = 2;
}

/* One group a CTA: the need smallest (key, slot) of its list, by byte digits
 * from the window's highest varying one. */
__global__ void __launch_bounds__(kThreads) k_rsel_pick(Sel S) {
  __shared__ uint32_t h[256];
  __shared__ uint64_t s_prefix;
  __shared__ int64_t s_need, s_slot;
  __shared__ uint32_t s_same;
  const int32_t g = blockIdx.x;
  const SelGroup G = S.g[g];
  const int64_t n = S.g[g + 1].start - G.start;
  if (G.k <= 0 || G.k >= n) return;
  const int64_t m = (int64_t)S.listed[g], need = G.k - (int64_t)S.below[g];
  if (need < 0 || need > m || m > G.cap) {
    if (threadIdx.x == 0) atomicOr(S.err, 1);
    return;
  }
  if (need == 0) return;
  const SelKey* L = S.list + G.list;
  if (threadIdx.x == 0) {
    s_prefix = 0;
    s_need = need;
    s_same = 0xffffffffu;
  }
  int shift = 64 - __clzll((long long)(G.hi - G.lo));
  shift = shift > 8 ? shift - 8 : 0;
  uint64_t fixed = 0; /* digits fixed so far: keys (less lo) that match s_prefix in the bits of `fixed` */
  __syncthreads();
  for (;;) {
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t prefix = s_prefix;
    for (int64_t q = threadIdx.x; q < m; q += blockDim.x) {
      const uint64_t v = L[q].key - G.lo;
      if ((v & fixed) == prefix) atomicAdd(&h[(v >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int64_t want = s_need;
      int d = 0;
      while (d < 255 && want > (int64_t)h[d]) want -= h[d++];
      s_need = want;
      s_prefix = prefix | (uint64_t)d << shift;
      s_same = h[d];
    }
    __syncthreads();
    fixed |= 255ULL << shift;
    if (s_same == 1 || shift == 0) break;
    shift = shift > 8 ? shift - 8 : 0;
  }
  /* the threshold's digits are s_prefix; of the s_same keys that share them
   * the s_need smallest are taken: all, unless whole keys are equal, when the
   * slots decide */
  const uint64_t prefix = s_prefix;
  if ((uint64_t)s_need < s_same) {
    for (int64_t q = threadIdx.x; q < m; q += blockDim.x) {
      if (((L[q].key - G.lo) & fixed) != prefix) continue;
      int64_t rank = 0;
      for (int64_t p = 0; p < m; ++p)
        rank += ((L[p].key - G.lo) & fixed) == prefix && L[p].slot < L[q].slot ? 1 : 0;
      if (rank == s_need - 1) s_slot = L[q].slot;
    }
  } else if (threadIdx.x == 0) {
    s_slot = INT64_MAX;
  }
  __syncthreads();
  for (int64_t q = threadIdx.x; q < m; q += blockDim.x) {
    const uint64_t v = (L[q].key - G.lo) & fixed;
    if (v < prefix || (v == prefix && L[q].slot <= s_slot)) atomicOr(&S.bits[L[q].slot >> 5], 1u << (L[q].slot & 31));
  }
}

__global__ void __launch_bounds__(kThreads) k_rsel_mark(const uint32_t* __restrict__ bits, lpg_columns c, int action, int64_t count) {
  const int64_t words = (count + 31) / 32, stride = (int64_t)gridDim.x * (kThreads / 32);
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int64_t w = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); w < words; w += stride)
    if (bits[w] >> lane & 1u) sel_apply(c, action, w * 32 + lane);
}

#define CKI(x)                                                                              \
  do {                                                                                      \
    cudaError_t e_ = (x);                                                                   \
    if (e_ != cudaSuccess) return lpg_ops_fail(LPG_ERR_CUDA, "init: %s", cudaGetErrorString(e_)); \
  } while (0)

/* A thread's workspace on a device, kept for its next call: a small table's
 * initialisation is five calls of some 50 us of kernels each, and an
 * allocation with its free costs 0.2 ms (the stream-ordered pool, which gives
 * its memory back at every synchronisation, the same).  4 MB at most a thread
 * and device, freed when the thread ends.  A call has its stream finish
 * before it returns, so the next one may use any stream.  All memory is
 * allocated and freed in stream order: cudaFree would wait for every stream's
 * kernels, of which a program may have a whole run queued. */
constexpr size_t kWorkBytes = 4 << 20, kTableBytes = 1 << 18;
struct Workspace {
  int device;
  uint8_t* dev;
  std::vector<uint8_t> host; /* the tables, as they go up */
};
struct Workspaces {
  std::vector<Workspace> all;
  ~Workspaces() {
    int device = 0;
    const bool known = cudaGetDevice(&device) == cudaSuccess;
    for (auto& w : all)
      if (cudaSetDevice(w.device) == cudaSuccess) cudaFreeAsync(w.dev, nullptr);
    if (known) cudaSetDevice(device);
  }
  Workspace* get(cudaStream_t st) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return nullptr;
    for (auto& w : all)
      if (w.device == device) return &w;
    Workspace w{device, nullptr, std::vector<uint8_t>(kTableBytes)};
    if (cudaMallocAsync((void**)&w.dev, kWorkBytes, st) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    all.push_back(std::move(w));
    return &all.back();
  }
};
thread_local Workspaces t_workspaces;

/* A call's device scratch: tables first, which go up with one copy
 * (ready()), then buffers, in the thread's workspace as far as it reaches and
 * allocated beyond. */
struct Scratch {
  cudaStream_t st;
  std::vector<void*> ptrs;
  Workspace* w;
  size_t used = 0, sent = 0, taken = kTableBytes;
  explicit Scratch(cudaStream_t s) : st(s), w(t_workspaces.get(s)) {}
  ~Scratch() {
    for (void* p : ptrs) cudaFreeAsync(p, st);
    cudaStreamSynchronize(st);
  }
  template <class T>
  int alloc(T** out, size_t n) {
    const size_t bytes = (n ? n : 1) * sizeof(T), room = (bytes + 255) & ~(size_t)255;
    if (w && taken + room <= kWorkBytes) {
      *out = (T*)(w->dev + taken);
      taken += room;
      return 0;
    }
    if (cudaMallocAsync((void**)out, bytes, st) != cudaSuccess) {
      cudaGetLastError();
      return lpg_ops_fail(LPG_ERR_NOMEM, "init: device scratch of %zu bytes", bytes);
    }
    ptrs.push_back(*out);
    return 0;
  }
  template <class T>
  int upload(T** out, const std::vector<T>& v) {
    const size_t bytes = v.size() * sizeof(T), room = (bytes + 255) & ~(size_t)255;
    if (!w || used + room > kTableBytes) {
      const int rc = alloc(out, v.size());
      if (rc) return rc;
      if (cudaMemcpyAsync(*out, v.data(), bytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return lpg_ops_fail(LPG_ERR_CUDA, "init: upload");
      return 0;
    }
    *out = (T*)(w->dev + used);
    if (bytes) memcpy(w->host.data() + used, v.data(), bytes);
    used += room;
    return 0;
  }
  /* before a kernel that reads what was uploaded */
  int ready() {
    if (used > sent &&
        cudaMemcpyAsync(w->dev + sent, w->host.data() + sent, used - sent, cudaMemcpyHostToDevice, st) != cudaSuccess)
      return lpg_ops_fail(LPG_ERR_CUDA, "init: upload");
    sent = used;
    return 0;
  }
};

int grid_for(int64_t n, int per_block) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int64_t want = (n + per_block - 1) / per_block;
  int64_t cap = (int64_t)(sms > 0 ? sms : 152) * 8;
  if (want > cap) want = cap;
  return (int)(want > 0 ? want : 1);
}

int select_k(Scratch& sc, cudaStream_t st, const lpg_columns& c, uint64_t seed, uint32_t purpose, int action,
             const std::vector<int64_t>& start, const std::vector<int64_t>& k, int64_t count) {
  const int32_t G = (int32_t)k.size();
  bool any = false;
  for (int32_t g = 0; g < G; ++g) any = any || (k[g] > 0 && start[g + 1] > start[g]);
  if (!any) return 0;
  Sel S{};
  S.seed = seed;
  S.purpose = purpose;
  S.n_groups = G;
  std::vector<SelGroup> groups(G + 1);
  const size_t words = (size_t)(count + 31) / 32;
  unsigned long long* counters; /* then the bits */
  int rc = sc.alloc(&counters, 2 * (size_t)G + 2 + (words + 1) / 2);
  if (rc) return rc;
  S.bits = reinterpret_cast<uint32_t*>(counters + 2 * (size_t)G + 2);
  S.below = counters;
  S.listed = counters + G;
  S.err = reinterpret_cast<int*>(counters + 2 * (size_t)G);
  for (double wide = 7.0;; wide *= 8.0) {
    int64_t total = 0;
    for (int32_t g = 0; g < G; ++g) {
      SelGroup& q = groups[g];
      const int64_t n = start[g + 1] - start[g];
      q = SelGroup{start[g], k[g], 0, ~0ULL, total, 0};
      if (k[g] <= 0 || k[g] >= n) continue;
      const double dn = (double)n, dk = (double)k[g], sd = std::sqrt(dk * (dn - dk) / dn) + 1.0;
      const double lo = (dk - wide * sd) / dn, hi = (dk + wide * sd) / dn;
      if (lo > 0.0) q.lo = (uint64_t)(lo * 18446744073709551616.0);
      if (hi < 1.0) q.hi = (uint64_t)(hi * 18446744073709551616.0);
      const double cap = (2.0 * wide + 8.0) * sd + 64.0;
      q.cap = cap < dn ? (int64_t)cap : n;
      total += q.cap;
    }
    groups[G] = SelGroup{start[G], 0, 0, 0, total, 0};
    SelGroup* d_groups;
    if ((rc = sc.upload(&d_groups, groups)) || (rc = sc.alloc(&S.list, (size_t)total)) || (rc = sc.ready())) return rc;
    S.g = d_groups;
    CKI(cudaMemsetAsync(counters, 0, sizeof(unsigned long long) * (2 * (size_t)G + 1), st));
    k_rsel_pass<<<grid_for(count, kTile), kThreads, 0, st>>>(S, count);
    k_rsel_pick<<<G, kThreads, 0, st>>>(S);
    CKI(cudaGetLastError());
    int h_err = 0;
    CKI(cudaMemcpyAsync(&h_err, S.err, sizeof(int), cudaMemcpyDeviceToHost, st));
    CKI(cudaStreamSynchronize(st));
    if (!h_err) break;
    if (wide > 1e12) return lpg_ops_fail(LPG_ERR_INTERNAL, "init: a selection window cannot miss every key");
  }
  k_rsel_mark<<<grid_for(count, kThreads * 4), kThreads, 0, st>>>(S.bits, c, action, count);
  CKI(cudaGetLastError());
  return 0;
}

/* Timers and heterogeneity by the FP32 kernels where the parameters have an
 * FP32 form (lpg_init_fast.cuh); the parts done are taken out of *parts.
 * The line is the form's own range: a lognormal that hardly varies would
 * put every draw beside the same whole day or FP32 step, all of them unsure
 * (2e7 slots at sigma 0: 26 ms against 22 in FP64 alone).  Small tables
 * take it too (16385 slots: 0.34 ms against 0.81). */
int fill_fast(Scratch& sc, cudaStream_t st, const lpg_init_desc& d, const SlotArgs& A, const lpg_columns& c,
              uint32_t* parts) {
  if (d.capacity <= 0) return 0;
  FiExact X{};
  X.seed = d.seed;
  X.capacity = d.capacity;
  X.c = c;
  const int grid = grid_for(d.capacity, FI_TILE), fix_grid = grid_for(d.capacity, FI_FIX_TILE);
  if (*parts & LPG_INIT_TIMERS) {
    const lpg_dist dist[3] = {d.dur_exp, d.dur_inf, d.t_to_paralysis};
    FiTimers F{};
    bool ok = true;
    int rc = 0;
    for (int b = 0; b < 3 && ok; ++b) {
      std::vector<uint64_t> thr;
      ok = fi_dist_of(dist[b], &F.d[b], &thr);
      if (ok && !thr.empty()) {
        uint64_t* p;
        if ((rc = sc.upload(&p, thr))) return rc;
        F.d[b].n_thr = (int32_t)thr.size();
        F.d[b].thr = p;
      }
    }
    if (ok) {
      if ((rc = sc.ready())) return rc;
      F.seed = d.seed;
      F.capacity = d.capacity;
      F.et = c.exposure_timer;
      F.it = c.infection_timer;
      F.pt = c.paralysis_timer;
      k_init_timers_fast<<<grid, FI_THREADS, 0, st>>>(F);
      X.k_exp = A.k_exp;
      X.k_inf = A.k_inf;
      X.k_par = A.k_par;
      X.e1 = A.e1;
      X.e2 = A.e2;
      X.i1 = A.i1;
      X.i2 = A.i2;
      X.p1 = A.p1;
      X.p2 = A.p2;
      k_init_fix<false><<<fix_grid, FI_THREADS, 0, st>>>(X);
      CKI(cudaGetLastError());
      *parts &= ~(uint32_t)LPG_INIT_TIMERS;
    }
  }
  if ((*parts & LPG_INIT_HETEROGENEITY) && A.het && A.sigma > 0.01 && A.sigma < 4.0 && A.scale < 1e6) {
    static const FiTables* host = fi_tables(); /* constants, formed once */
    FiTables* tab;
    int rc = sc.upload(&tab, std::vector<FiTables>(1, *host));
    if (!rc) rc = sc.ready();
    if (rc) return rc;
    FiHet H{d.seed, d.capacity, fi_pair(A.mu), fi_pair(A.sigma), fi_pair(A.rho), fi_pair(A.srho), fi_pair(A.scale),
            tab, c.acq_risk_multiplier, c.daily_infectivity};
    k_init_het_fast<<<grid, FI_THREADS, 0, st>>>(H);
    X.mu = A.mu;
    X.sigma = A.sigma;
    X.rho = A.rho;
    X.srho = A.srho;
    X.scale = A.scale;
    k_init_fix<true><<<fix_grid, FI_THREADS, 0, st>>>(X);
    CKI(cudaGetLastError());
    *parts &= ~(uint32_t)LPG_INIT_HETEROGENEITY;
  }
  return 0;
}

}  // namespace

extern "C" double lpg_init_mean_infectivity(uint64_t seed, double r0, lpg_dist dur_inf) {
  lpg_stream s;
  lpg_stream_init(&s, seed, LPG_P_INIT_MEANINF, 0, 0, 0);
  double sum = 0.0;
  for (int j = 0; j < 1000; ++j) sum = sum + lpg_dist_sample(&s, dur_inf.kind, dur_inf.p1, dur_inf.p2);
  return r0 / (sum / 1000.0);
}

extern "C" int lpg_init_columns(const lpg_init_desc* d, uint32_t parts, const lpg_columns* cols, void* stream) {
  if (!d || !cols) return lpg_ops_fail(LPG_ERR_ARG, "init: null argument");
  const int32_t n = d->n_nodes;
  if (n < 1 || n > 32767) return lpg_ops_fail(LPG_ERR_ARG, "init: n_nodes %d out of range", n);
  if (d->count < 0 || d->capacity < d->count || d->capacity >= (int64_t)0xFFFFFFF0LL)
    return lpg_ops_fail(LPG_ERR_ARG, "init: count %lld / capacity %lld", (long long)d->count, (long long)d->capacity);
  if (!d->node_pop) return lpg_ops_fail(LPG_ERR_ARG, "init: node_pop is required");
  std::vector<int64_t> start(n + 1, 0);
  for (int i = 0; i < n; ++i) {
    if (d->node_pop[i] < 0) return lpg_ops_fail(LPG_ERR_ARG, "init: node_pop[%d] is negative", i);
    start[i + 1] = start[i] + d->node_pop[i];
  }
  if (start[n] != d->count) return lpg_ops_fail(LPG_ERR_ARG, "init: node_pop sums to %lld, count is %lld",
                                                (long long)start[n], (long long)d->count);
  const lpg_columns& c = *cols;
  auto need = [&](uint32_t part, std::initializer_list<const void*> ptrs, const char* what) -> int {
    if (!(parts & part)) return 0;
    for (const void* p : ptrs)
      if (!p) return lpg_ops_fail(LPG_ERR_ARG, "init: %s needs its columns", what);
    return 0;
  };
  int rc = 0;
  if ((rc = need(LPG_INIT_BASE, {c.disease_state, c.node_id, c.strain, c.potentially_paralyzed, c.paralyzed,
                                 c.ipv_protected, c.chronically_missed}, "BASE")) ||
      (rc = need(LPG_INIT_MISSED, {c.chronically_missed}, "MISSED")) ||
      (rc = need(LPG_INIT_TIMERS, {c.exposure_timer, c.infection_timer, c.paralysis_timer}, "TIMERS")) ||
      (rc = need(LPG_INIT_IMMUNITY, {c.disease_state, d->immune_k}, "IMMUNITY")) ||
      (rc = need(LPG_INIT_PREVALENCE, {c.disease_state, d->prev_k}, "PREVALENCE")) ||
      (rc = need(LPG_INIT_HETEROGENEITY, {c.acq_risk_multiplier, c.daily_infectivity}, "HETEROGENEITY")) ||
      (rc = need(LPG_INIT_AGES, {c.date_of_birth, d->age_lo_days, d->age_hi_days, d->age_weight}, "AGES")) ||
      (rc = need(LPG_INIT_DEATHS, {c.date_of_birth, c.date_of_death, d->km_cumdeaths}, "DEATHS")) ||
      (rc = need(LPG_INIT_RI, {c.date_of_birth, c.ri_timer}, "RI")))
    return rc;
  cudaStream_t st = (cudaStream_t)stream;
  Scratch sc(st);
  SlotArgs A{};
  A.seed = d->seed;
  A.count = d->count;
  A.capacity = d->capacity;
  A.n_nodes = n;
  if (parts & LPG_INIT_BASE) {
    int64_t* d_start;
    if ((rc = sc.upload(&d_start, start))) return rc;
    A.node_start = d_start;
  }
  A.k_exp = d->dur_exp.kind;
  A.e1 = d->dur_exp.p1;
  A.e2 = d->dur_exp.p2;
  A.k_inf = d->dur_inf.kind;
  A.i1 = d->dur_inf.p1;
  A.i2 = d->dur_inf.p2;
  A.k_par = d->t_to_paralysis.kind;
  A.p1 = d->t_to_paralysis.p1;
  A.p2 = d->t_to_paralysis.p2;
  if (parts & LPG_INIT_HETEROGENEITY) {
    /* model.py:839-851: lognormal risk with mean 1 and variance risk_mult_var;
     * infectivity mean r0 / mean(dur_inf(1000)), at least 1e-10 */
    const double var = d->risk_mult_var;
    if (!(var >= 0.0) || !std::isfinite(var)) return lpg_ops_fail(LPG_ERR_ARG, "init: risk_mult_var %g", var);
    A.het = d->heterogeneity != 0;
    A.mu = std::log(1.0 / std::sqrt(var + 1.0));
    A.sigma = std::sqrt(std::log(var + 1.0));
    A.rho = 2.0 * std::sin(LPG_PI * d->corr_risk_inf / 6.0);
    if (!(std::fabs(A.rho) <= 1.0)) return lpg_ops_fail(LPG_ERR_ARG, "init: corr_risk_inf %g", d->corr_risk_inf);
    A.srho = std::sqrt(1.0 - A.rho * A.rho);
    const double mean = lpg_init_mean_infectivity(d->seed, d->r0, d->dur_inf);
    A.scale = mean > 1e-10 ? mean : 1e-10;
  }
  if (parts & LPG_INIT_AGES) {
    const int nb = d->n_age_bins;
    if (nb < 1) return lpg_ops_fail(LPG_ERR_ARG, "init: no age bins");
    std::vector<int64_t> cum(nb);
    std::vector<int32_t> lo(d->age_lo_days, d->age_lo_days + nb), hi(d->age_hi_days, d->age_hi_days + nb);
    int64_t acc = 0;
    for (int b = 0; b < nb; ++b) {
      if (d->age_weight[b] < 0 || hi[b] <= lo[b]) return lpg_ops_fail(LPG_ERR_ARG, "init: age bin %d", b);
      acc += d->age_weight[b];
      cum[b] = acc;
    }
    if (acc <= 0) return lpg_ops_fail(LPG_ERR_ARG, "init: age weights sum to 0");
    A.n_bins = nb;
    int64_t* dc;
    int32_t *dl, *dh;
    if ((rc = sc.upload(&dc, cum)) || (rc = sc.upload(&dl, lo)) || (rc = sc.upload(&dh, hi))) return rc;
    A.age_cum = dc;
    A.age_lo = dl;
    A.age_hi = dh;
  }
  if (parts & LPG_INIT_DEATHS) {
    if (d->km_len < 1) return lpg_ops_fail(LPG_ERR_ARG, "init: empty km table");
    std::vector<int64_t> km(d->km_cumdeaths, d->km_cumdeaths + d->km_len);
    int64_t* dk;
    if ((rc = sc.upload(&dk, km))) return rc;
    A.km = dk;
    A.km_len = d->km_len;
    A.km_max_year = d->km_max_year;
  }
  uint32_t slot_parts =
      parts & (LPG_INIT_BASE | LPG_INIT_TIMERS | LPG_INIT_HETEROGENEITY | LPG_INIT_AGES | LPG_INIT_DEATHS | LPG_INIT_RI);
  if ((rc = fill_fast(sc, st, *d, A, c, &slot_parts))) return rc;
  if ((slot_parts & LPG_INIT_BASE) && d->capacity > 0) {
    const void* ps[] = {c.disease_state, c.node_id, c.strain, c.potentially_paralyzed, c.paralyzed, c.ipv_protected,
                        c.chronically_missed};
    bool wide = true;
    for (const void* q : ps) wide = wide && ((uintptr_t)q & 15u) == 0;
    if ((rc = sc.ready())) return rc;
    k_init_base<<<grid_for(d->capacity, kThreads * 16), kThreads, 0, st>>>(A, c, wide);
    CKI(cudaGetLastError());
    slot_parts &= ~(uint32_t)LPG_INIT_BASE;
  }
  const uint32_t dates = slot_parts & (LPG_INIT_AGES | LPG_INIT_DEATHS | LPG_INIT_RI);
  if (dates && d->capacity > 0) {
    if ((rc = sc.ready())) return rc;
    k_init_dates<<<grid_for(d->capacity, kThreads * 8), kThreads, 0, st>>>(A, c, dates);
    CKI(cudaGetLastError());
    slot_parts &= ~dates;
  }
  if (slot_parts && d->capacity > 0) {
    if ((rc = sc.ready())) return rc;
    k_init_slots<<<grid_for(d->capacity, kThreads * 8), kThreads, 0, st>>>(A, c, slot_parts);
    CKI(cudaGetLastError());
  }
  const std::vector<int64_t> all = {0, d->count};
  if ((parts & LPG_INIT_MISSED) && d->count > 0) {
    if ((rc = select_k(sc, st, c, d->seed, LPG_P_INIT_MISSED, 0, all, {d->missed_k}, d->count))) return rc;
  }
  if ((parts & LPG_INIT_IMMUNITY) && d->count > 0) {
    std::vector<int64_t> k(d->immune_k, d->immune_k + n);
    if ((rc = select_k(sc, st, c, d->seed, LPG_P_INIT_IMMUNE, 1, start, k, d->count))) return rc;
  }
  if ((parts & LPG_INIT_PREVALENCE) && d->count > 0) {
    if (d->prev_per_node) {
      std::vector<int64_t> k(d->prev_k, d->prev_k + n);
      rc = select_k(sc, st, c, d->seed, LPG_P_INIT_PREV, 2, start, k, d->count);
    } else {
      rc = select_k(sc, st, c, d->seed, LPG_P_INIT_PREV, 2, all, {d->prev_k[0]}, d->count);
    }
    if (rc) return rc;
  }
  CKI(cudaStreamSynchronize(st));
  return LPG_OK;
}
