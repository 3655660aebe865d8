// lev_grid.cuh -- grid-resident engine for mid-sized networks and batches.
// Included once, from lev_engine.cu.
//
// Networks whose CTAs all fit on the device at once (one cooperative launch,
// co-residency guaranteed by the launch) are stepped n times in ONE launch: a
// single network, or a batch, whose networks step independently of one
// another:
//   * CTA b of a network owns its rows [b*R, b*R + R), R = 64, 128 or 256, with
//     four, two or one lanes per row (lev_split.cuh); its SELL-32 slices
//     (col|delay, weights) stay in shared memory and its rows' node state in
//     registers for the whole launch;
//   * the delay ring stays in global memory, which at these sizes is
//     L2-resident: each step writes theta(t+1) of the CTA's rows to ring slot
//     t+1 through L2.  Gathers may hit L1: a CTA acquires the arrivals of every
//     step (ld.acquire.gpu, which drops the SM's L1 lines) before it gathers
//     phases of that step, so no line outlives a rewrite of its slot.  Within a
//     step a 32-byte sector (two nodes, four slots) serves three gathers of a
//     tile; through L2 only, N = 10^5, k = 20 took 8.4 us per step against 7.6;
//   * every CTA publishes its part of (sum cos, sum sin) of a step, and every
//     CTA adds all parts in the order of leviathan_kernel.cu:198-263, so all
//     CTAs of a network compute the same r and gain (see grid_kernel);
//   * an arrival counter per network orders the ring's phases;
//   * an attached hub monitor is fed by the network's CTA 0.
// Arithmetic and summation order are those of step_kernel: results are
// bitwise the same as stepping with step_kernel.
//
// Every wait is bounded (GridWait, 2 s by default): on a timeout
// the CTA writes 1 to the error flag (mapped host memory), leaves the step
// loop and writes nothing back; the host reports the error.

#pragma once

#include "lev_split.cuh"

namespace lev {

struct GridArgs {
  const NetDesc *nets;
  NetState *st;
  const int2 *map;  // per CTA (network, CTA within the network); null: one network
  const int *row_ptr;
  const long long *sl_off;
  const int *sl_len;
  const uint32_t *sl_cd;
  float *sl_w;
  float *theta;
  float *theta_hat;
  const float *omega;
  float *omega_hat;
  float *ring;
  float2 *wsum;      // per network [4][8 * tiles] sums, at 32 * part_off; kNoSum at launch
  unsigned *bar;     // per network arrival counter, zero at launch, kGridBarPitch apart
  HubMonitor *hubs;  // observes hub phases after every step of hubs->net, or null
  int early;         // no delay is 0: wait for barrier t after step t+1's edges
  int *err;          // error flag (mapped host memory)
  GridWait wait;     // bound of the barrier waits
  float *r_hist;     // [r_cap][num_nets] (row rpos + k), or null
  int r_cap;
  int num_nets;
  int n_steps;
  int edge_cap;      // SELL entries per CTA the shared memory was sized for
  int sum_cap;       // sums staged per CTA the shared memory was sized for (R < 256)
  float dt;
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Grid barrier, split in two.  Arrive: every thread of the CTA calls it
// after its writes; thread 0 adds one arrival with release semantics, which
// (after the CTA barrier) publishes the writes of the whole CTA.
__device__ __forceinline__ void grid_arrive(unsigned *bar) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}

// Wait: every thread of the CTA calls it; thread 0 waits (acquire) until
// `target` arrivals (plus gw.extra), at most gw.ns.  Returns false after a
// timeout, in every thread.
__device__ __forceinline__ bool grid_wait(unsigned *bar, unsigned target, int *err, int *s_ok,
                                          const GridWait &gw) {
  if (threadIdx.x == 0) {
    const unsigned long long t0 = global_ns();
    while (ld_acquire_gpu(bar) < target + gw.extra) {
      if (global_ns() - t0 > gw.ns) {
        *reinterpret_cast<volatile int *>(err) = 1;
        *s_ok = 0;
        break;
      }
    }
  }
  __syncthreads();
  return *reinterpret_cast<volatile int *>(s_ok) != 0;
}

// Waits like grid_wait, but one lane only; returns false after a timeout.
__device__ __forceinline__ bool grid_poll(unsigned *bar, unsigned target, const GridWait &gw) {
  const unsigned long long t0 = global_ns();
  while (ld_acquire_gpu(bar) < target + gw.extra)
    if (global_ns() - t0 > gw.ns) return false;
  return true;
}

// A sum that has not been published yet: a NaN pattern that no published sum
// has (grid_publish changes it into another NaN).
constexpr unsigned kNoSum = 0xffffffffu;

__device__ __forceinline__ uint4 ld_relaxed_gpu4(const void *p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint2 ld_relaxed_gpu2(const void *p) {
  uint2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void grid_publish(float2 *p, float2 v) {
  unsigned x = __float_as_uint(v.x), y = __float_as_uint(v.y);
  if (x == kNoSum) x = 0x7fffffffu;
  if (y == kNoSum) y = 0x7fffffffu;
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void grid_unpublish(float2 *p) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %1};" ::"l"(p), "r"(kNoSum) : "memory");
}

// Waits, at most gw.ns, until all sums of a step are published and adds them
// up, one warp; returns false, in every lane, after a timeout.
//   BLOCKS: `n` sums of whole 256-node blocks; lane l takes blocks l, l+32, ...
//           and adds them in the order of leviathan_kernel.cu:242-263.
//   else:   `n` sums of 32-row slices (an even number), read as 16-byte pairs
//           in memory order, staged in s_sum (zeros up to 8 per block) and
//           formed into blocks with the reference's second-level tree
//           (:216-233) first.
template <bool BLOCKS>
__device__ __forceinline__ bool grid_sums(const float2 *buf, int n, int nblocks, int lane,
                                          const GridWait &gw, float2 *s_sum, float2 *out) {
  const unsigned mask = 0xffffffffu;
  const unsigned long long t0 = global_ns();
  float sum_cos = 0.0f, sum_sin = 0.0f;
  constexpr int K = 8;  // loads in flight per lane
  const int items = BLOCKS ? n : n / 2;
  for (int base = 0; base < items; base += 32 * K) {
    uint4 v[K];
    for (;;) {
      bool ready = gw.extra == 0;
#pragma unroll
      for (int j = 0; j < K; ++j) {
        const int i = base + 32 * j + lane;
        v[j] = make_uint4(0u, 0u, 0u, 0u);
        if (i < items) {
          if (BLOCKS) {
            const uint2 t = ld_relaxed_gpu2(buf + i);
            v[j].x = t.x;
            v[j].y = t.y;
          } else {
            v[j] = ld_relaxed_gpu4(buf + 2 * i);
          }
        }
      }
#pragma unroll
      for (int j = 0; j < K; ++j) {
        ready = ready && v[j].x != kNoSum && v[j].y != kNoSum;
        if (!BLOCKS) ready = ready && v[j].z != kNoSum && v[j].w != kNoSum;
      }
      if (__all_sync(mask, ready)) break;
      if (__any_sync(mask, global_ns() - t0 > gw.ns)) return false;
    }
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = base + 32 * j + lane;
      if (i >= items) continue;
      if (BLOCKS) {
        sum_cos += __uint_as_float(v[j].x);
        sum_sin += __uint_as_float(v[j].y);
      } else {
        reinterpret_cast<uint4 *>(s_sum)[i] = v[j];
      }
    }
  }
  if (!BLOCKS) {
    __syncwarp();
    for (int b = lane; b < nblocks; b += 32) {
      float vc[8], vs[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 t = reinterpret_cast<const float4 *>(s_sum)[4 * b + i];
        vc[2 * i] = t.x;
        vs[2 * i] = t.y;
        vc[2 * i + 1] = t.z;
        vs[2 * i + 1] = t.w;
      }
      sum_cos += block_tree8(vc);
      sum_sin += block_tree8(vs);
    }
    __syncwarp();
  }
#pragma unroll
  for (int off = 16; off > 0; off /= 2) {
    sum_cos += __shfl_down_sync(mask, sum_cos, off);
    sum_sin += __shfl_down_sync(mask, sum_sin, off);
  }
  *out = make_float2(sum_cos, sum_sin);
  return true;
}

constexpr unsigned kSumsSleep = 400;  // ns, of a sums warp before its first poll
constexpr int kGridBarPitch = 32;  // arrival counters of two networks share no 128-byte line
constexpr int kGridThreads = 256 + 32;  // eight warps on rows, one for the other CTAs

// grid_kernel for at most `minb` CTAs per SM: two (with an order warp where a
// row has several lanes) or three.
__host__ __device__ constexpr bool grid_order_warp(int R, int minb) { return minb == 2 && R < 256; }
// Most entries of a lane in flight together: twelve at one lane per row where
// the registers allow it, but not with the accurate sine and cosine (N = 2*10^4,
// accurate, R = 256: eight 7.4 us per recorded step, twelve 9.9).
__host__ __device__ constexpr int grid_walk_max(int math, int R, int minb) {
  return math == 0 && R == 256 && minb == 2 ? 12 : 8;
}
__host__ __device__ constexpr int grid_threads(int R, int minb) {
  return grid_order_warp(R, minb) ? 256 + 64 : kGridThreads;
}

// Barrier of a CTA whose warps run different code.
template <int THREADS = kGridThreads>
__device__ __forceinline__ void cta_barrier() {
  asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
}

// One warp publishes its CTA's sums of step `step` from the warps' parts and
// clears those of step-2 for step+2.
template <int R>
__device__ __forceinline__ void grid_publish_part(float2 *wsum, int step, int nblocks, int nsum,
                                                  int cta, int lane, const float2 *s_part) {
  constexpr int LPR = 256 / R;
  constexpr int count = R == 256 ? 1 : R / 32;
  const int at = cta * count + lane;
  if (lane >= count || at >= nsum) return;
  float2 v;
  if (R == 256) {
    float vc[8], vs[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      vc[i] = s_part[i].x;
      vs[i] = s_part[i].y;
    }
    v = make_float2(block_tree8(vc), block_tree8(vs));
  } else {
    v = split_slice_sum<LPR>(s_part + LPR * lane);
  }
  grid_publish(wsum + (step & 3) * 8 * nblocks + at, v);
  grid_unpublish(wsum + ((step + 2) & 3) * 8 * nblocks + at);
}

// shared memory layout (bytes, from the dynamic base):
//   sums   float2 [8 * blocks of the largest network]  (R < 256)
//   sloff, sllen  int [R/32]
//   cd     uint32 [edge_cap]  (order of lev_split.cuh)
//   w      float  [edge_cap]
// R: rows per CTA, 64, 128 or 256, with LPR = 256 / R lanes per row.
//
// What bounds a step is a chain of L2 round trips (about 600 cycles each).
// With the CTA's first warp doing both its rows' edges and the exchange, at N =
// 10^4 (R = 64) a step took 6,990 cycles: edges 2,070, waiting for the counter
// 960, reading the sums 2,130, integrate 620, and 1,190 in the release fence
// of the arrival, one after the other.  So the exchange has warps of its own,
// and the sums carry their own "published" mark: they go out without waiting
// for the fence, which only the ring phases need.  The sums warp publishes and
// collects the sums, the order warp pays the fence, arrives and waits for the
// others' arrivals.  With R = 256 and in grids of more than two CTAs per SM
// (MINB = 3, 72 registers) one warp does both, in that order: there the rows'
// gathers bound the step.  With R = 256 and MINB = 2 a lane has up to twelve
// entries in flight instead of eight and 96 registers: at 72 the long rows'
// loads come one after the other.  us per step, MINB = 3 / 2: N = 3,000, k = 32
// 6.9 / 4.5; 37,800, k = 32 7.1 / 5.1; 5*10^4, k = 8 3.6 / 3.2; 5*10^4, k = 20 5.6 /
// 5.3; 64 networks of 500 to 2,000 rows, k up to 32 12.0 / 7.0.
//
// Order of one step s:
//   edge warps            | sums warp                 | order warp
//   predictor, edges      | wait for the sums of s-1; | fence and arrive for s-1
//                         | r, g of step s            |
//   ------------------------------- barrier A: g ----------------------------
//   integrate, slot s+1   |                           | wait for every arrival s-1
//   ------------------------------- barrier B: warp parts -------------------
//   (step s+1)            | publish the sums of s,    | fence, arrive for s
//                         | clear those of s-2        |
// Gathers of step s+1 read slots <= s (no zero delay), whose phases arrivals
// s-1 ordered before barrier B of step s.  The integrate of step s overwrites
// the slot that the gathers of step s-1 read last; those CTAs have published
// the sums of s-1, which follow from the gathered values.  Sums of s live in
// buffer s mod 4; a CTA clears its part of buffer (s+2) mod 4, the sums of s-2,
// once all sums of s-1 have shown that nobody still reads them, and its arrival
// s+1 orders the clearing before anybody looks for the sums of s+2 there (in
// step s+3).  With zero delays step s gathers slot s, and the wait for arrivals
// s-1 comes before the edges (barrier C).
//
// Every wait for arrivals comes late, when they have mostly come: polling from
// the arrival on holds up the arrivals themselves, and every acquire drops the
// L1 lines the gathers live on.  The sums warp sleeps before its first poll for
// the same reason.  Measured per step (us), edges and exchange in one warp / one
// exchange warp / two: N = 6,000, k = 20 (R = 64) - / 2.37 / 2.11; N = 10^4 (64)
// 3.5 / 2.62 / 2.46; N = 18,900 (128) - / 3.17 / 2.85; N = 10^5 (256) - / 7.6 /
// 8.8 (two steps per launch: 13.1).
template <int MATH, int R, int MINB>
__global__ void __launch_bounds__(grid_threads(R, MINB), MINB) grid_kernel(const GridArgs a) {
  constexpr int LPR = 256 / R;
  constexpr bool ORDER = grid_order_warp(R, MINB);
  constexpr int kThreads = grid_threads(R, MINB);
  constexpr int kUM = grid_walk_max(MATH, R, MINB);
  constexpr int nslices = R / 32;
  constexpr bool kBlocks = R == 256;  // a CTA closes its 256-node block itself
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_g;
  __shared__ int s_ok;
  __shared__ float2 s_part[8];

  const int2 me = a.map ? a.map[blockIdx.x] : make_int2(0, (int)blockIdx.x);
  const NetDesc nd = a.nets[me.x];
  const int cta = me.y;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool edges = warp < 8;
  const SplitLane sl = split_lane<LPR>(tid & 255);
  const int N = nd.N, bsi = nd.bsi, Np = nd.Np;
  const int row0 = cta * R;
  const int row = row0 + sl.rloc;
  const bool live = edges && row < N;
  const unsigned G = (unsigned)((N + R - 1) / R);
  const int nblocks = nd.ntiles;
  unsigned *bar = a.bar + kGridBarPitch * me.x;
  float2 *wsum = a.wsum + 32 * (long long)nd.part_off;  // four buffers of 8 * nblocks
  // sums published per step: blocks, or slices up to the last whole block
  const int nsum = kBlocks ? nblocks : min(8 * nblocks, (int)G * nslices);

  float2 *s_sum = reinterpret_cast<float2 *>(smem);
  int *sloff = reinterpret_cast<int *>(s_sum + a.sum_cap);
  int *sllen = sloff + nslices;
  uint32_t *s_cd = reinterpret_cast<uint32_t *>(sllen + nslices);
  float *s_w = reinterpret_cast<float *>(s_cd + a.edge_cap);

  // ---- load this CTA's part of the network --------------------------------
  const long long sl0 = nd.slice_base + row0 / 32;
  const int my_slices = max(0, min(nslices, (N - row0 + 31) / 32));
  const long long ebase = my_slices ? a.sl_off[sl0] : 0;
  for (int s = tid; s < nslices; s += blockDim.x) {
    sloff[s] = s < my_slices ? (int)(a.sl_off[sl0 + s] - ebase) : 0;
    sllen[s] = s < my_slices ? a.sl_len[sl0 + s] : 0;
  }
  for (int k = tid; k < a.sum_cap; k += blockDim.x) s_sum[k] = make_float2(0.0f, 0.0f);
  if (tid == 0) s_ok = 1;
  __syncthreads();
  split_for_entries<LPR>(sloff, sllen, my_slices, [&](int at, int e) {
    s_cd[at] = a.sl_cd[ebase + e];
    s_w[at] = a.sl_w[ebase + e];
  });
  const long long gi = nd.node_off + row;
  int deg = 0;
  float th = 0.0f, thh = 0.0f, om = 0.0f, omh = 0.0f;  // alike in the row's lanes
  if (live) {
    th = a.theta[gi];
    thh = a.theta_hat[gi];
    om = a.omega[gi];
    omh = a.omega_hat[gi];
    const int *rp = a.row_ptr + nd.rp_off + row;
    deg = rp[1] - rp[0];
  }
  const NetState ns = a.st[me.x];
  int cur = ns.cur;
  float g = ns.g;
  float *ring = a.ring + nd.ring_off;
  const float dt = a.dt;
  __syncthreads();

  // a timeout of one of the exchange warps: all warps read the flag after
  // barrier A, and it is only written between B and A
  auto stopped = [&]() { return *reinterpret_cast<volatile int *>(&s_ok) == 0; };
  auto give_up = [&]() {
    if (lane == 0) {
      *reinterpret_cast<volatile int *>(a.err) = 1;
      *reinterpret_cast<volatile int *>(&s_ok) = 0;
    }
    __syncwarp();
  };
  // the phases of the first `steps` steps of every CTA are in the ring
  auto phases_of = [&](int steps) -> bool {
    const bool ok = lane != 0 || grid_poll(bar, (unsigned)steps * G, a.wait);
    return __all_sync(0xffffffffu, ok);
  };
  auto arrive = [&]() {
    if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
  };
  if (edges) {
    const int len = sllen[sl.ws], base = sloff[sl.ws];
    for (int step = 0; step < a.n_steps; ++step) {
      if (step > 0 && !a.early) cta_barrier<kThreads>();  // C
      // ---- predictor; edges -------------------------------------------------------
      float eps = 0.0f;
      auto predictor = [&]() -> EdgeParams {
        eps = sinf(wrap_pm_pi(th - thh));
        thh = thh + dt * omh;
        omh = omh + nd.kappa_w * dt * eps;
        return {dt, nd.eta, nd.lam, __fmaf_rn(-nd.gamma, fabsf(eps), 1.0f), nd.w_min, nd.w_max};
      };
      auto gather = [&](uint32_t word) {
        return __ldca(ring + ring_pos_word(word, cur, bsi, Np));
      };
      float local_sum;
      if constexpr (ORDER) {
        // the edges are on the step's critical path: the predictor runs while
        // the first gathers are in flight
        local_sum = split_walk<MATH, LPR>(s_cd + base, s_w + base, len, deg, sl, th, predictor,
                                          gather);
      } else {
        const EdgeParams ep = predictor();
        local_sum =
            split_walk<MATH, LPR, kUM>(s_cd + base, s_w + base, len, deg, sl, th, ep, gather);
      }
      if (step > 0) {
        cta_barrier<kThreads>();  // A
        if (stopped()) break;
        g = s_g;
      }
      // ---- integrate --------------------------------------------------------------
      int nxt = cur + 1;
      if (nxt == bsi) nxt = 0;
      float my_cos = 0.0f, my_sin = 0.0f;
      if (live) {
        float inc = dt * (om + g * local_sum - nd.alpha * eps);
        float x = th + inc;
        x = wrap_0_2pi(x);
        if (!isfinite(x)) x = 0.0f;
        th = x;
        if (sl.q == 0) __stcg(ring + ring_pos(nxt, row, Np), x);
        lev_sincos<MATH>(x, &my_sin, &my_cos);
      }
      const float2 part = split_warp_sum<LPR>(my_cos, my_sin);
      if (lane == 0) s_part[warp] = part;
      cur = nxt;
      cta_barrier<kThreads>();  // B
    }
  } else {
    // what the two exchange warps do; one warp does both where there is no
    // order warp
    const bool sums = warp == 8, order = warp == 9 || !ORDER;
    const float inv_N = 1.0f / (float)N;
    float r = ns.r;
    // CTA 0 feeds an attached hub monitor
    const bool observe = order && a.hubs && a.hubs->net == me.x && cta == 0;
    HubWarp hub;
    if (observe) hub.open(a.hubs);
    // r and g after `steps` steps of this launch (lane 0); false after a timeout
    auto close_step = [&](int steps) -> bool {
      float2 s;
      if (!grid_sums<kBlocks>(wsum + ((steps - 1) & 3) * 8 * nblocks, nsum, nblocks, lane, a.wait,
                              s_sum, &s))
        return false;
      r = order_parameter(s.x, s.y, inv_N);
      if (nd.ctrl) g = gain_controller(g, r, dt, nd);
      if (lane == 0) {
        s_g = g;
        if (cta == 0 && a.r_hist) {
          const int k = ns.rpos + steps - 1;
          if (k < a.r_cap) a.r_hist[(long long)k * a.num_nets + me.x] = r;
        }
      }
      return true;
    };
    bool ok = true, go_on = true;
    float hub_phase = 0.0f;
    for (int step = 0; step < a.n_steps; ++step) {
      if (step > 0) {
        if (!a.early) {
          if (order && !phases_of(step)) give_up();
          cta_barrier<kThreads>();  // C
        }
        if (sums) {
          if (ORDER) __nanosleep(kSumsSleep);
          if (!close_step(step)) give_up();
        }
        cta_barrier<kThreads>();  // A
        if (stopped()) {
          go_on = false;
          break;
        }
        // a timeout here is reported after B (see stopped)
        if (order && a.early) ok = phases_of(step);
        if (observe) hub_phase = __ldcg(ring + ring_pos(cur, hub.node, Np));
      }
      cur = (cur + 1 == bsi) ? 0 : cur + 1;
      cta_barrier<kThreads>();  // B
      if (!ok) give_up();
      if (sums) {
        grid_publish_part<R>(wsum, step, nblocks, nsum, cta, lane, s_part);
        __syncwarp();
      }
      if (order) arrive();
      if (observe && step > 0) hub.observe(hub_phase);
    }
    // CTA 0 closes the last step
    if (go_on && ok && a.n_steps > 0 && cta == 0) {
      if (observe) {
        if (!phases_of(a.n_steps)) give_up();
        hub.observe(__ldcg(ring + ring_pos(cur, hub.node, Np)));
        hub.close(a.n_steps);
      }
      if (sums) {
        if (!close_step(a.n_steps)) {
          give_up();
        } else if (lane == 0) {
          NetState o = ns;
          o.g = g;
          o.r = r;
          o.cur = cur;
          o.rbuf = (int)((ns.rbuf + (long long)a.n_steps) % (nd.max_delay + 1));
          o.t = ns.t + a.n_steps;
          o.rpos = ns.rpos + a.n_steps;
          o.ticket = 0u;
          a.st[me.x] = o;
        }
      }
    }
  }
  __syncthreads();
  if (*reinterpret_cast<volatile int *>(&s_ok) == 0) return;  // timeout: the host reports it
  // ---- write the state back -------------------------------------------------
  if (live && sl.q == 0) {
    a.theta[gi] = th;
    a.theta_hat[gi] = thh;
    a.omega_hat[gi] = omh;
  }
  split_for_entries<LPR>(sloff, sllen, my_slices,
                         [&](int at, int e) { a.sl_w[ebase + e] = s_w[at]; });
}

}  // namespace lev
