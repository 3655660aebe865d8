// lev_split.cuh -- SELL-32 rows worked by one, two or four lanes, their entries
// in shared memory: the edge walk shared by the cluster- and grid-resident
// kernels.
//
// With one lane per row a small network leaves the SMs waiting on instruction
// latency; four lanes per row give four times the warps.  What the split costs
// is the row sum, which has to be formed in CSR order with the reference's
// multiply-adds.  Lane q of a row takes U consecutive entries per chunk of
// LPR * U, and the running sum is handed from lane to lane: LPR times (U
// multiply-adds and one shuffle) per chunk.  Fetching every term to the row's
// first lane instead took two shuffles and a select per entry: N = 1000, k = 20
// on 16 CTAs 2.83 us per step, 1.93 us with this walk and the row order below.
//
// Rows to lanes: warp c of the LPR warps of a 32-row slice holds rows c, c + LPR,
// c + 2 LPR, ... of the slice, lane LPR * m + q being lane q of row c + LPR * m.
// The reference's shuffle tree over 32 rows (leviathan_kernel.cu:198-214) adds
// rows 16, 8, 4, 2, 1 apart: its first levels then stay in the warp and the
// last log2(LPR) are additions over the slice's warps.
//
// Entries in shared memory: entry (k, l) of a slice lies at
// 32k + ((l + (k / U mod LPR)) mod 32), so the 32 lanes of a warp read 32
// different banks; with the global layout 32k + l the lanes of a row met on
// one bank.
#pragma once

#include <type_traits>

#include "lev_kernels.cuh"

namespace lev {

constexpr unsigned long long kGridWaitNs = 2000000000ull;  // default wait limit

// Bound of every wait on other CTAs of a launch.  `extra` is 0 in normal use;
// a positive value makes each wait expect that many arrivals more than the
// grid makes, so the first wait runs out after `ns` -- the timeout path can
// then be exercised by a test without faulting or hanging the GPU.
struct GridWait {
  unsigned long long ns;  // limit of one wait, globaltimer nanoseconds
  unsigned extra;
  unsigned pad;
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Entries per lane and chunk for slices of `len` entries per row: as few
// chunks as entries of at most UM per lane allow, of equal size (an empty
// entry costs the instructions of a full one).  With one lane per row the
// order in shared memory does not depend on it.
template <int LPR, int UM = 8>
__device__ __forceinline__ int split_unroll(int len) {
  static_assert(UM == 8 || LPR == 1, "");
  const int chunks = max((len + UM * LPR - 1) / (UM * LPR), 1);
  return max((len + LPR * chunks - 1) / (LPR * chunks), 1);
}

struct SplitLane {
  int q;     // lane of the row, 0 .. LPR - 1
  int l;     // row within its 32-row slice
  int ws;    // slice within the CTA
  int rloc;  // row within the CTA
  int lead;  // first lane of the row
};
template <int LPR>
__device__ __forceinline__ SplitLane split_lane(int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  SplitLane s;
  s.q = lane & (LPR - 1);
  s.lead = lane & ~(LPR - 1);
  s.l = (warp & (LPR - 1)) + s.lead;  // c + LPR m
  s.ws = warp / LPR;
  s.rloc = 32 * s.ws + s.l;
  return s;
}

// Copies between the slices' global order and the shared order above, one
// warp per 32 entries: f(position in shared memory, entry index from the
// CTA's first entry).
template <int LPR, class F>
__device__ __forceinline__ void split_for_entries(const int *sloff, const int *sllen, int nslices,
                                                  F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int s = 0; s < nslices; ++s) {
    const int off = sloff[s], len = sllen[s];
    const int u = split_unroll<LPR>(len);
    for (int k = warp; k < len; k += nwarps)
      f(off + 32 * k + ((lane + ((k / u) & (LPR - 1))) & 31), off + 32 * k + lane);
  }
}

// The row's walk (csr_physics_kernel, leviathan_kernel.cu:126-165) over cd /
// w, the slice's entries in shared memory; gather(word) returns the delayed
// phase and keep(k, weight) sees the new weight of the row's entry k.  `params`
// is the row's EdgeParams, or a function that returns them, run once while the
// first chunk's gathers are in flight (it may do the row's predictor there).
// Returns the row's coupling sum in all its lanes.  Entries past the
// row's degree enter the sum as 0 * sin(0 - th): a zero, or a NaN in a row
// whose phase is not finite and whose step sets it to 0 whatever the sum.
template <int MATH, int LPR, int U, class Params, class Gather, class Keep>
__device__ __forceinline__ float split_walk_u(const uint32_t *cd, float *w, int len, int deg,
                                              const SplitLane &sl, float th, Params &params,
                                              Gather gather, Keep keep) {
  constexpr bool kGiven = std::is_same<Params, const EdgeParams>::value;
  EdgeParams ep;
  if constexpr (kGiven) ep = params;
  const unsigned mask = 0xffffffffu;
  const int lq = (sl.l + sl.q) & 31;
  float local_sum = 0.0f;
  if constexpr (!kGiven)
    if (len == 0) params();
  for (int kb = 0; kb < len; kb += LPR * U) {  // len: the slice's, warp-uniform
    const int k0 = kb + U * sl.q;
    const int at = 32 * k0 + lq;
    uint32_t p[U];
    float wv[U], dj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const bool in = k0 + u < deg;
      p[u] = in ? cd[at + 32 * u] : 0u;
      wv[u] = in ? w[at + 32 * u] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) dj[u] = (k0 + u < deg) ? gather(p[u]) : 0.0f;
    if constexpr (!kGiven)
      if (kb == 0) ep = params();
#pragma unroll
    for (int u = 0; u < U; ++u) dj[u] -= th;
    float sn[U], cs[U];
    wrap_sincos_group<MATH>(dj, sn, cs);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const float wn = edge_weight(ep, cs[u], wv[u]);
      if (k0 + u < deg) {
        w[at + 32 * u] = wn;
        keep(k0 + u, wn);
      }
    }
#pragma unroll
    for (int ph = 0; ph < LPR; ++ph) {
#pragma unroll
      for (int u = 0; u < U; ++u) local_sum = __fmaf_rn(wv[u], sn[u], local_sum);
      if (LPR > 1) local_sum = __shfl_sync(mask, local_sum, sl.lead + ph);
    }
  }
  return local_sum;
}

template <int MATH, int LPR, int UM = 8, class Params, class Gather, class Keep>
__device__ __forceinline__ float split_walk(const uint32_t *cd, float *w, int len, int deg,
                                            const SplitLane &sl, float th, Params &params,
                                            Gather gather, Keep keep) {
  switch (split_unroll<LPR, UM>(len)) {  // warp-uniform
    case 1: return split_walk_u<MATH, LPR, 1>(cd, w, len, deg, sl, th, params, gather, keep);
    case 2: return split_walk_u<MATH, LPR, 2>(cd, w, len, deg, sl, th, params, gather, keep);
    case 3: return split_walk_u<MATH, LPR, 3>(cd, w, len, deg, sl, th, params, gather, keep);
    case 4: return split_walk_u<MATH, LPR, 4>(cd, w, len, deg, sl, th, params, gather, keep);
    case 5: return split_walk_u<MATH, LPR, 5>(cd, w, len, deg, sl, th, params, gather, keep);
    case 6: return split_walk_u<MATH, LPR, 6>(cd, w, len, deg, sl, th, params, gather, keep);
    case 7: return split_walk_u<MATH, LPR, 7>(cd, w, len, deg, sl, th, params, gather, keep);
    case 8: return split_walk_u<MATH, LPR, 8>(cd, w, len, deg, sl, th, params, gather, keep);
  }
  if constexpr (UM > 8) {
    static_assert(UM == 12, "");
    switch (split_unroll<LPR, UM>(len)) {
      case 9: return split_walk_u<MATH, LPR, 9>(cd, w, len, deg, sl, th, params, gather, keep);
      case 10: return split_walk_u<MATH, LPR, 10>(cd, w, len, deg, sl, th, params, gather, keep);
      case 11: return split_walk_u<MATH, LPR, 11>(cd, w, len, deg, sl, th, params, gather, keep);
    }
    return split_walk_u<MATH, LPR, 12>(cd, w, len, deg, sl, th, params, gather, keep);
  }
  return 0.0f;  // not reached
}
template <int MATH, int LPR, int UM = 8, class Params, class Gather>
__device__ __forceinline__ float split_walk(const uint32_t *cd, float *w, int len, int deg,
                                            const SplitLane &sl, float th, Params &params,
                                            Gather gather) {
  return split_walk<MATH, LPR, UM>(cd, w, len, deg, sl, th, params, gather, [](int, float) {});
}

// The warp's part of the 32-row tree: rows 16 down to LPR apart; lane 0 holds
// the sum of the warp's rows.  The lanes of a row hold equal values.
template <int LPR>
__device__ __forceinline__ float2 split_warp_sum(float c, float s) {
  const unsigned mask = 0xffffffffu;
#pragma unroll
  for (int off = 16; off >= LPR; off /= 2) {
    c += __shfl_down_sync(mask, c, off);
    s += __shfl_down_sync(mask, s, off);
  }
  return make_float2(c, s);
}
// ... and its last levels over the slice's LPR warps.
template <int LPR>
__device__ __forceinline__ float2 split_slice_sum(const float2 *p) {
  if (LPR == 1) return p[0];
  if (LPR == 2) return make_float2(p[0].x + p[1].x, p[0].y + p[1].y);
  return make_float2((p[0].x + p[2].x) + (p[1].x + p[3].x),
                     (p[0].y + p[2].y) + (p[1].y + p[3].y));
}

// The observations of a hub monitor over the steps of one launch (hub_observe,
// once per step), by one warp: lane i watches hub i.  Indices and the previous
// state stay in registers and the counters take fire-and-forget additions, so
// an observation costs the warp one ring load, issued early by the caller, and
// a few instructions.
struct HubWarp {
  HubMonitor *hm;
  unsigned long long *counts, *totals;
  int num_hubs, node, prev;
  __device__ __forceinline__ void open(HubMonitor *m) {
    const int lane = threadIdx.x & 31;
    hm = m;
    counts = m->counts;
    totals = m->totals;
    num_hubs = m->num_hubs;
    prev = m->prev;
    node = m->hub[lane < num_hubs ? lane : 0];
  }
  __device__ __forceinline__ void observe(float phase) {
    const int lane = threadIdx.x & 31;
    float x = fmodf(phase, 6.2831853f);
    if (x < 0) x += 6.2831853f;
    const int state =
        (int)__ballot_sync(0xffffffffu, lane < num_hubs && x > 3.1415926f);
    const int S = 1 << num_hubs;
    if (lane == 0 && prev >= 0 && prev < S) {
      atomicAdd(counts + (long long)prev * S + state, 1ull);
      atomicAdd(totals + prev, 1ull);
    }
    prev = state;
  }
  __device__ __forceinline__ void close(int observed) {
    if ((threadIdx.x & 31) == 0) {
      hm->prev = prev;
      hm->observed += observed;
    }
  }
};

// r of (sum cos, sum sin) (leviathan_kernel.cu:262), the squares fused as nvcc
// fuses them there; inv_N = 1 / N.
__device__ __forceinline__ float order_parameter(float sum_cos, float sum_sin, float inv_N) {
  return sqrtf(__fmaf_rn(sum_cos, sum_cos, __fmul_rn(sum_sin, sum_sin))) * inv_N;
}

}  // namespace lev
