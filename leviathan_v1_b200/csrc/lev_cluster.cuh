// lev_cluster.cuh -- cluster-resident engine for small networks.  Included
// once, from lev_engine.cu.
//
// A network of up to 16 x 1024 nodes whose edges, node state and delay ring
// fit in the shared memory of one thread-block cluster (up to 16 CTAs, one per
// SM, 227 KB each) is stepped n times in ONE launch:
//   * CTA r of the cluster owns rows [r*R, r*R + R), R a multiple of 32, one
//     thread per row; its SELL-32 slices (col|delay, weights), its node state
//     and its rows of every ring slot live in its shared memory;
//   * a delayed phase of a node owned by another CTA is read from that CTA's
//     shared memory (distributed shared memory, cluster.map_shared_rank);
//   * one cluster barrier per step, split into an arrival after step t's
//     ring write and warp sums and a wait before step t+1's integrate (which
//     needs g(t+1) and overwrites ring slot t+2 = t-max_delay, read by step
//     t).  Without zero delays step t+1's gathers read slots <= t, ordered by
//     the barrier of step t-1, so the predictor and the edge work of step t+1
//     run while the barrier of step t completes; with zero delays the wait
//     comes before the gathers (with max_delay+2 ring slots, reads and the
//     write of one step never touch the same slot);
//   * each warp's shuffle-tree (sum cos, sum sin) of its 32 rows goes to a
//     double-buffered array in CTA 0; after the barrier every CTA forms the
//     256-node block sums from eight warp sums with the arithmetic of the
//     reference's block tree (leviathan_kernel.cu:198-233) and reduces the
//     blocks in the order of :242-263, so all CTAs compute the same r and
//     gain without a second barrier.  A 256-node block may thus span CTAs,
//     and a small network spreads over up to 16 SMs.
// Arithmetic and summation order are those of step_kernel: results are
// bitwise the same as stepping with step_kernel.

#include <cooperative_groups.h>

#include "lev_split.cuh"

namespace lev {

constexpr int kClusterMax = 16;     // CTAs per cluster (non-portable size)
constexpr int kClusterRowsMax = 1024;
constexpr int kClusterWarpsMax = kClusterMax * kClusterRowsMax / 32;  // 512

// Sum of one 256-node block from its eight warp sums v[0..7], with the
// arithmetic of the reference's second-level tree (leviathan_kernel.cu:
// 216-233: warp 0 takes the eight warp sums in lanes 0-7, zeros elsewhere,
// then shuffle-down adds at offsets 16, 8, 4, 2, 1): the first two levels add
// zeros (which turns -0 into +0), then (v0+v4, ...), then pairs, then one.
__device__ __forceinline__ float block_tree8(const float *v) {
  float z[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) z[i] = __fadd_rn(__fadd_rn(v[i], 0.0f), 0.0f);
  const float a0 = __fadd_rn(z[0], z[4]), a1 = __fadd_rn(z[1], z[5]);
  const float a2 = __fadd_rn(z[2], z[6]), a3 = __fadd_rn(z[3], z[7]);
  return __fadd_rn(__fadd_rn(a0, a2), __fadd_rn(a1, a3));
}

// r of one step from the warp sums wsum[nwarps_blocks * 8] (one warp: lane l
// adds blocks l, l+32, ..., then the shuffle tree), as final_reduce_r_kernel
// (leviathan_kernel.cu:242-263) over the reference's block partials.
__device__ __forceinline__ float2 cluster_sums(const float2 *wsum, int nblocks, int lane) {
  float sum_cos = 0.0f, sum_sin = 0.0f;
  for (int b = lane; b < nblocks; b += 32) {
    float vc[8], vs[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = wsum[b * 8 + i];
      vc[i] = v.x;
      vs[i] = v.y;
    }
    sum_cos += block_tree8(vc);
    sum_sin += block_tree8(vs);
  }
  const unsigned mask = 0xffffffffu;
#pragma unroll
  for (int off = 16; off > 0; off /= 2) {
    sum_cos += __shfl_down_sync(mask, sum_cos, off);
    sum_sin += __shfl_down_sync(mask, sum_sin, off);
  }
  return make_float2(sum_cos, sum_sin);
}

struct ClusterArgs {
  const NetDesc *net;
  NetState *st;
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
  float *r_hist;  // [n] (row rpos + k), or null
  HubMonitor *hubs;  // observes hub phases after every step, or null (cluster_split_kernel)
  int r_cap;
  int n_steps;
  int R;          // rows per CTA (a power of two, 32 .. 1024)
  int lgR;        // log2(R)
  int edge_cap;   // SELL entries per CTA the shared memory was sized for
  int early;      // no delay is 0: wait for step t's barrier after step t+1's edges
  int *err;       // error flag (mapped host memory) (cluster_split_kernel)
  GridWait wait;  // bound of the waits (cluster_split_kernel)
  float dt;
};

// Split cluster barrier (every thread of every CTA of the cluster): arrival
// with release semantics, wait with acquire semantics.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// shared memory layout (bytes, from the dynamic base):
//   wsum   float2 [2][kClusterWarpsMax]        warp sums (used in CTA 0)
//   sloff  int    [R/32]   slice start (relative to the CTA's first entry)
//   sllen  int    [R/32]
//   th, thh, om, omh  float [R]
//   ring   float  [bsi][R]
//   cd     uint32 [edge_cap]
//   w      float  [edge_cap]
// MAXR: largest rows per CTA of the instantiation (the register budget);
// U: edges per lane whose gathers are in flight together.
template <int MATH, int MAXR, int U>
__global__ void __launch_bounds__(MAXR, 1) cluster_kernel(const ClusterArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem[];

  const NetDesc nd = *a.net;
  const int rank = (int)cluster.block_rank();
  const int R = a.R;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int N = nd.N, bsi = nd.bsi, Np = nd.Np;
  const int row0 = rank * R;
  const int row = row0 + tid;
  const bool live = (tid < R) && (row < N);
  const int nslices = R / 32;

  float2 *wsum = reinterpret_cast<float2 *>(smem);
  int *sloff = reinterpret_cast<int *>(wsum + 2 * kClusterWarpsMax);
  int *sllen = sloff + nslices;
  float *s_th = reinterpret_cast<float *>(sllen + nslices);
  float *s_thh = s_th + R;
  float *s_om = s_thh + R;
  float *s_omh = s_om + R;
  float *s_ring = s_omh + R;
  uint32_t *s_cd = reinterpret_cast<uint32_t *>(s_ring + (size_t)bsi * R);
  float *s_w = reinterpret_cast<float *>(s_cd + a.edge_cap);

  // ---- load this CTA's part of the network --------------------------------
  const long long sl0 = nd.slice_base + row0 / 32;
  const int my_slices = max(0, min(nslices, (N - row0 + 31) / 32));
  const long long ebase = my_slices ? a.sl_off[sl0] : 0;
  long long eend = ebase;
  for (int s = tid; s < nslices; s += blockDim.x) {
    if (s < my_slices) {
      sloff[s] = (int)(a.sl_off[sl0 + s] - ebase);
      sllen[s] = a.sl_len[sl0 + s];
    } else {
      sloff[s] = 0;
      sllen[s] = 0;
    }
  }
  if (my_slices) eend = a.sl_off[sl0 + my_slices - 1] + 32LL * a.sl_len[sl0 + my_slices - 1];
  const int nent = (int)(eend - ebase);
  for (int k = tid; k < nent; k += blockDim.x) {
    s_cd[k] = a.sl_cd[ebase + k];
    s_w[k] = a.sl_w[ebase + k];
  }
  int deg = 0;
  if (live) {
    const long long gi = nd.node_off + row;
    s_th[tid] = a.theta[gi];
    s_thh[tid] = a.theta_hat[gi];
    s_om[tid] = a.omega[gi];
    s_omh[tid] = a.omega_hat[gi];
    const int *rp = a.row_ptr + nd.rp_off + row;
    deg = rp[1] - rp[0];
  }
  for (int s = 0; s < bsi; ++s)
    if (live) s_ring[(size_t)s * R + tid] = a.ring[nd.ring_off + ring_pos(s, row, Np)];
  NetState ns = *a.st;
  int cur = ns.cur, rbuf = ns.rbuf;
  float g = ns.g, r = ns.r;
  const int nblocks = (N + kTile - 1) / kTile;
  // warps past the network's last row contribute zero sums to their block
  if (rank == 0)
    for (int k = tid; k < 2 * kClusterWarpsMax; k += blockDim.x) wsum[k] = make_float2(0.0f, 0.0f);
  const float dt = a.dt;
  const float eta = nd.eta, gamma = nd.gamma, lam = nd.lam;
  const float w_min = nd.w_min, w_max = nd.w_max;
  const unsigned mask = 0xffffffffu;
  cluster.sync();

  float2 *wsum0 = cluster.map_shared_rank(wsum, 0);
  __shared__ float s_g;
  for (int step = 0; step < a.n_steps; ++step) {
    // with zero delays: step-1's barrier before the gathers
    if (step > 0 && !a.early) cluster_wait();
    // ---- predictor --------------------------------------------------------
    float th = 0.0f, eps = 0.0f;
    if (live) {
      th = s_th[tid];
      const float thh = s_thh[tid];
      const float wh = s_omh[tid];
      float diff = th - thh;
      diff = wrap_pm_pi(diff);
      eps = sinf(diff);
      s_thh[tid] = thh + dt * wh;
      s_omh[tid] = wh + nd.kappa_w * dt * eps;
    }
    const float my_eps = fabsf(eps);
    // ---- edges --------------------------------------------------------------
    float local_sum = 0.0f;
    if (warp < my_slices) {
      const int len = sllen[warp];
      const int base = sloff[warp] + lane;
      for (int k0 = 0; k0 < len; k0 += U) {
        uint32_t p[U];
        float wv[U], dj[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const bool in = k0 + u < deg;
          p[u] = in ? s_cd[base + 32 * (k0 + u)] : 0u;
          wv[u] = in ? s_w[base + 32 * (k0 + u)] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          int slot = cur - (int)(p[u] & 255u);
          slot += (slot < 0) ? bsi : 0;
          const int j = (int)(p[u] >> 8);
          const int owner = j >> a.lgR;
          const int loc = j & (R - 1);
          const float *src = (owner == rank) ? s_ring : cluster.map_shared_rank(s_ring, owner);
          dj[u] = src[(size_t)slot * R + loc];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (k0 + u < deg) {
            const float delayed_j = dj[u];
            float diff = delayed_j - th;
            diff = wrap_pm_pi(diff);
            float w = wv[u];
            float sin_diff, cos_diff;
            lev_sincos<MATH>(diff, &sin_diff, &cos_diff);
            local_sum += w * sin_diff;
            float dw = dt * (eta * cos_diff * (1.0f - gamma * my_eps) - lam * w);
            w += dw;
            if (!isfinite(w)) w = w_min;
            w = fmaxf(w_min, fminf(w_max, w));
            s_w[base + 32 * (k0 + u)] = w;
          }
        }
      }
    }
    // ---- r and gain of the previous step: warp 0 of every CTA reduces the
    // block partials (same order everywhere) and shares g with its CTA ----
    if (step > 0) {
      if (a.early) cluster_wait();
      if (warp == 0) {
        const float2 sums =
            cluster_sums(wsum0 + ((step - 1) & 1) * kClusterWarpsMax, nblocks, lane);
        const float sum_cos = sums.x, sum_sin = sums.y;
        if (lane == 0) {
          float inv_N = 1.0f / (float)N;
          r = sqrtf(sum_cos * sum_cos + sum_sin * sum_sin) * inv_N;
          if (nd.ctrl) g = gain_controller(g, r, dt, nd);
          s_g = g;
          if (rank == 0 && a.r_hist) {
            const int k = ns.rpos + step - 1;
            if (k < a.r_cap) a.r_hist[k] = r;
          }
        }
      }
      __syncthreads();
      g = s_g;
    }
    // ---- integrate ----------------------------------------------------------
    int nxt = cur + 1;
    if (nxt == bsi) nxt = 0;
    float my_cos = 0.0f, my_sin = 0.0f;
    if (live) {
      float inc = dt * (s_om[tid] + g * local_sum - nd.alpha * eps);
      float x = th + inc;
      x = wrap_0_2pi(x);
      if (!isfinite(x)) x = 0.0f;
      s_th[tid] = x;
      s_ring[(size_t)nxt * R + tid] = x;
      lev_sincos<MATH>(x, &my_sin, &my_cos);
    }
    // ---- warp sums of (cos, sin), first level of the block tree
    // (leviathan_kernel.cu:198-214), to CTA 0 ------------------------------
#pragma unroll
    for (int off = 16; off > 0; off /= 2) {
      my_cos += __shfl_down_sync(mask, my_cos, off);
      my_sin += __shfl_down_sync(mask, my_sin, off);
    }
    if (lane == 0)
      wsum0[(step & 1) * kClusterWarpsMax + row0 / 32 + warp] = make_float2(my_cos, my_sin);
    cur = nxt;
    rbuf = (rbuf + 1 == nd.max_delay + 1) ? 0 : rbuf + 1;
    cluster_arrive();
  }
  if (a.n_steps > 0) cluster_wait();
  // ---- r of the last step, then write the state back ------------------------
  if (a.n_steps > 0) {
    const float2 sums =
        cluster_sums(wsum0 + ((a.n_steps - 1) & 1) * kClusterWarpsMax, nblocks, lane);
    const float sum_cos = __shfl_sync(mask, sums.x, 0);
    const float sum_sin = __shfl_sync(mask, sums.y, 0);
    float inv_N = 1.0f / (float)N;
    r = sqrtf(sum_cos * sum_cos + sum_sin * sum_sin) * inv_N;
    if (nd.ctrl) g = gain_controller(g, r, dt, nd);
    if (rank == 0 && tid == 0) {
      if (a.r_hist) {
        const int k = ns.rpos + a.n_steps - 1;
        if (k < a.r_cap) a.r_hist[k] = r;
      }
      NetState o = ns;
      o.g = g;
      o.r = r;
      o.cur = cur;
      o.rbuf = rbuf;
      o.t = ns.t + a.n_steps;
      o.rpos = ns.rpos + a.n_steps;
      o.ticket = 0u;
      *a.st = o;
    }
  }
  if (live) {
    const long long gi = nd.node_off + row;
    a.theta[gi] = s_th[tid];
    a.theta_hat[gi] = s_thh[tid];
    a.omega_hat[gi] = s_omh[tid];
    for (int s = 0; s < bsi; ++s)
      a.ring[nd.ring_off + ring_pos(s, row, Np)] = s_ring[(size_t)s * R + tid];
  }
  for (int k = tid; k < nent; k += blockDim.x) a.sl_w[ebase + k] = s_w[k];
  // no CTA may leave while a peer can still read its shared memory
  cluster.sync();
}

// ---------------------------------------------------------------------------
// The cluster-resident step with four lanes per row (R up to 128; rows and
// entries to lanes as in lev_split.cuh) and a warp for the other CTAs.  Bitwise
// the results of cluster_kernel and step_kernel.
//
// A step is one latency chain (N = 1000: 16 CTAs of 64 rows, two warps per SM
// sub-core).  With every thread in the cluster barrier, 710 of a step's 3,800
// cycles went into the arrival, whose release waits for the remote stores of
// the sums, and 600 into the reduction.  So the exchange has a warp of its own,
// as in grid_kernel: it sends its CTA's slice sums to every CTA with st.async,
// which signals the receiver's mbarrier as the data lands and needs no answer,
// waits on its own mbarrier for those of all CTAs and reduces them, while the
// edge warps walk the next step's edges.
//
// Order of one step s (barriers A and B are the CTA's):
//   edge warps               | exchange warp
//   predictor, edges         | wait for all slice sums of s-1; r, g of step s
//   ------------------------ barrier A: g (before the edges with zero delays)
//   integrate, ring slot s+1 |
//   ------------------------ barrier B: warp parts
//   (step s+1)               | send the slice sums of s to every CTA
// With the sums goes an arrival with release semantics, which orders the CTA's
// phases of step s: gathers of step s+1 read slots <= s, and every CTA's arrival
// of step s-1 was among those that barrier A of step s waited for.  The integrate of step s
// overwrites the slot that the gathers of step s-1 read last; the CTAs that did
// have sent the sums of s-1, which follow from the gathered values.  Sums of s
// go to buffer s mod 2: whoever sends them has received all sums of s-1, whose
// senders had done with those of s-2.
// ---------------------------------------------------------------------------
constexpr int kSplitLPR = 4;  // lanes per row
constexpr int kSplitSlicesMax = kClusterMax * 128 / 32;  // 64: at most 8 blocks of 256 nodes

__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
// 8 bytes to another CTA's shared memory, counted by the mbarrier `bar` there.
__device__ __forceinline__ void st_cluster_async(uint32_t addr, float2 v, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(
          addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// An arrival at an mbarrier of the cluster that orders this CTA's writes before it.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar)
               : "memory");
}
// This phase's arrival, and the bytes it waits for.
__device__ __forceinline__ void mbar_expect(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
               "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}

// (sum cos, sum sin) from up to 64 slice sums (zero past the network), by one
// warp, in every lane: three shuffle levels close the 256-node blocks
// (block_tree8), and two more add the at most eight blocks in the order of
// final_reduce_r_kernel (leviathan_kernel.cu:242-263: lane b holds block b, the
// first two levels add zeros).
__device__ __forceinline__ float2 split_sums(const float2 *sums, int nslices, int lane) {
  const unsigned mask = 0xffffffffu;
  float c[2] = {0.0f, 0.0f}, s[2] = {0.0f, 0.0f};
#pragma unroll
  for (int grp = 0; grp < 2; ++grp) {
    if (32 * grp >= nslices) break;  // uniform
    const float2 a = sums[32 * grp + lane];
    float vc = __fadd_rn(__fadd_rn(a.x, 0.0f), 0.0f);
    float vs = __fadd_rn(__fadd_rn(a.y, 0.0f), 0.0f);
#pragma unroll
    for (int off = 4; off > 0; off /= 2) {
      vc += __shfl_down_sync(mask, vc, off);
      vs += __shfl_down_sync(mask, vs, off);
    }
    c[grp] = __fadd_rn(0.0f, vc);  // lanes 0, 8, 16, 24: blocks 4 grp + 0 .. 3
    s[grp] = __fadd_rn(0.0f, vs);
  }
  float sc = c[0] + c[1], ss = s[0] + s[1];
#pragma unroll
  for (int off = 16; off >= 8; off /= 2) {
    sc += __shfl_down_sync(mask, sc, off);
    ss += __shfl_down_sync(mask, ss, off);
  }
  return make_float2(__shfl_sync(mask, sc, 0), __shfl_sync(mask, ss, 0));
}

// shared memory (bytes, from the dynamic base):
//   sums   float2 [2][kSplitSlicesMax]   every CTA's copy of the slice sums
//   sloff, sllen  int [R/32]
//   ring   float  [bsi][R]
//   cd     uint32 [edge_cap], w float [edge_cap]   (order of lev_split.cuh)
// The wait is bounded (GridWait): on a timeout the CTA writes 1 to the error
// flag (mapped host memory), leaves the step loop and writes nothing back.
template <int MATH>
__global__ void __launch_bounds__(kSplitLPR * 128 + 32, 1)
    cluster_split_kernel(const ClusterArgs a) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) unsigned long long s_mbar[2];
  __shared__ float2 s_part[kSplitLPR * 128 / 32];
  __shared__ float s_g;
  __shared__ int s_ok;

  const NetDesc nd = *a.net;
  const int rank = (int)cluster.block_rank();
  const int C = (int)cluster.num_blocks();
  const int R = a.R;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthreads = blockDim.x;  // 4R + 32
  const bool edges = tid < kSplitLPR * R;
  const SplitLane sl = split_lane<kSplitLPR>(edges ? tid : lane);
  const int N = nd.N, bsi = nd.bsi, Np = nd.Np;
  const int row0 = rank * R;
  const int row = row0 + sl.rloc;
  const bool live = edges && row < N;
  const int nslices = R / 32;
  auto cta_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory"); };

  float2 *s_sums = reinterpret_cast<float2 *>(smem);
  int *sloff = reinterpret_cast<int *>(s_sums + 2 * kSplitSlicesMax);
  int *sllen = sloff + nslices;
  float *s_ring = reinterpret_cast<float *>(sllen + nslices);
  uint32_t *s_cd = reinterpret_cast<uint32_t *>(s_ring + (size_t)bsi * R);
  float *s_w = reinterpret_cast<float *>(s_cd + a.edge_cap);

  // ---- load this CTA's part of the network --------------------------------
  const long long sl0 = nd.slice_base + row0 / 32;
  const int my_slices = max(0, min(nslices, (N - row0 + 31) / 32));
  const long long ebase = my_slices ? a.sl_off[sl0] : 0;
  for (int s = tid; s < nslices; s += nthreads) {
    sloff[s] = s < my_slices ? (int)(a.sl_off[sl0 + s] - ebase) : 0;
    sllen[s] = s < my_slices ? a.sl_len[sl0 + s] : 0;
  }
  for (int k = tid; k < 2 * kSplitSlicesMax; k += nthreads) s_sums[k] = make_float2(0.0f, 0.0f);
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(s_mbar);
  if (tid == 0) {
    s_ok = 1;
    mbar_init(mbar, (unsigned)C + 1u);  // every CTA, and this one's expected bytes
    mbar_init(mbar + 8, (unsigned)C + 1u);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  split_for_entries<kSplitLPR>(sloff, sllen, my_slices, [&](int at, int e) {
    s_cd[at] = a.sl_cd[ebase + e];
    s_w[at] = a.sl_w[ebase + e];
  });
  int deg = 0;
  float th = 0.0f, thh = 0.0f, om = 0.0f, omh = 0.0f;  // alike in the row's four lanes
  if (live) {
    const long long gi = nd.node_off + row;
    th = a.theta[gi];
    thh = a.theta_hat[gi];
    om = a.omega[gi];
    omh = a.omega_hat[gi];
    const int *rp = a.row_ptr + nd.rp_off + row;
    deg = rp[1] - rp[0];
    for (int s = sl.q; s < bsi; s += kSplitLPR)
      s_ring[(size_t)s * R + sl.rloc] = a.ring[nd.ring_off + ring_pos(s, row, Np)];
  }
  const NetState ns = *a.st;
  int cur = ns.cur;
  float g = ns.g;
  const float dt = a.dt;
  const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(s_ring);
  auto phase = [&](int j, int slot) {
    const uint32_t at = ring_addr + 4u * (unsigned)(slot * R + (j & (R - 1)));
    return ld_cluster(cluster_addr(at, j >> a.lgR));
  };
  cluster.sync();

  if (edges) {
    const int len = sllen[sl.ws], base = sloff[sl.ws];
    for (int step = 0; step < a.n_steps; ++step) {
      if (step > 0 && !a.early) {
        cta_sync();  // A, before the gathers of slot `step`
        if (*reinterpret_cast<volatile int *>(&s_ok) == 0) break;
      }
      // ---- predictor ----------------------------------------------------------
      const float eps = sinf(wrap_pm_pi(th - thh));
      thh = thh + dt * omh;
      omh = omh + nd.kappa_w * dt * eps;
      // ---- edges ----------------------------------------------------------------
      const EdgeParams ep = {dt, nd.eta, nd.lam, __fmaf_rn(-nd.gamma, fabsf(eps), 1.0f),
                             nd.w_min, nd.w_max};
      const float local_sum =
          split_walk<MATH, kSplitLPR>(s_cd + base, s_w + base, len, deg, sl, th, ep,
                                      [&](uint32_t word) {
            const unsigned s0 = (unsigned)(cur - (int)(word & 255u));
            return phase((int)(word >> 8), (int)min(s0, s0 + (unsigned)bsi));
          });
      if (step > 0) {
        if (a.early) {
          cta_sync();  // A
          if (*reinterpret_cast<volatile int *>(&s_ok) == 0) break;
        }
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
        if (sl.q == 0) s_ring[(size_t)nxt * R + sl.rloc] = x;
        lev_sincos<MATH>(x, &my_sin, &my_cos);
      }
      // ---- this warp's part of the slice sums (leviathan_kernel.cu:198-214) -------
      const float2 part = split_warp_sum<kSplitLPR>(my_cos, my_sin);
      if (lane == 0) s_part[warp] = part;
      cur = nxt;
      cta_sync();  // B
    }
  } else {
    const float inv_N = 1.0f / (float)N;
    const int all_slices = 8 * nd.ntiles;
    const unsigned bytes = (unsigned)(C * nslices) * 8u;
    float r = ns.r;
    // lane c sends to CTA c
    const int to = lane < C ? lane : 0;
    const uint32_t sums_to = cluster_addr(
        (uint32_t)__cvta_generic_to_shared(s_sums + row0 / 32), to);
    const uint32_t mbar_to = cluster_addr(mbar, to);
    // CTA 0 feeds an attached hub monitor
    const bool observe = a.hubs && rank == 0;
    HubWarp hub;
    if (observe) hub.open(a.hubs);
    // r and g after `steps` steps of this launch, alike in every lane; false
    // after a timeout
    auto close_step = [&](int steps) -> bool {
      const int b = (steps - 1) & 1;
      const unsigned parity = (unsigned)((steps - 1) >> 1) & 1u;
      const unsigned long long t0 = global_ns();
      while (a.wait.extra || !__all_sync(0xffffffffu, mbar_try_wait(mbar + 8 * b, parity)))
        if (__any_sync(0xffffffffu, global_ns() - t0 > a.wait.ns)) return false;
      const float2 sums = split_sums(s_sums + b * kSplitSlicesMax, all_slices, lane);
      r = order_parameter(sums.x, sums.y, inv_N);
      if (nd.ctrl) g = gain_controller(g, r, dt, nd);
      if (lane == 0) {
        s_g = g;
        if (rank == 0 && a.r_hist) {
          const int k = ns.rpos + steps - 1;
          if (k < a.r_cap) a.r_hist[k] = r;
        }
      }
      return true;
    };
    auto give_up = [&]() {
      if (lane == 0) {
        *reinterpret_cast<volatile int *>(a.err) = 1;
        *reinterpret_cast<volatile int *>(&s_ok) = 0;
      }
      __syncwarp();
    };
    bool ok = true;
    for (int step = 0; step < a.n_steps; ++step) {
      float hub_phase = 0.0f;
      if (step > 0) {
        ok = close_step(step);
        if (!ok) give_up();
        cta_sync();  // A
        if (!ok) break;
        if (observe) hub_phase = phase(hub.node, cur);
      }
      if (lane == 0) mbar_expect(mbar + 8 * (step & 1), bytes);
      cur = (cur + 1 == bsi) ? 0 : cur + 1;
      cta_sync();  // B
      if (lane < C) mbar_arrive_cluster(mbar_to + 8u * (unsigned)(step & 1));
      for (int s = 0; s < nslices; ++s) {
        const float2 v = split_slice_sum<kSplitLPR>(s_part + kSplitLPR * s);
        if (lane < C)
          st_cluster_async(sums_to + 8u * (unsigned)((step & 1) * kSplitSlicesMax + s), v,
                           mbar_to + 8u * (unsigned)(step & 1));
      }
      __syncwarp();
      if (observe && step > 0) hub.observe(hub_phase);
    }
    // the last step: every CTA waits for its sums (they land in its memory)
    if (ok && a.n_steps > 0) {
      ok = close_step(a.n_steps);
      if (!ok) give_up();
      if (ok && rank == 0) {
        if (lane == 0) {
          NetState o = ns;
          o.g = g;
          o.r = r;
          o.cur = cur;
          o.rbuf = (int)((ns.rbuf + (long long)a.n_steps) % (nd.max_delay + 1));
          o.t = ns.t + a.n_steps;
          o.rpos = ns.rpos + a.n_steps;
          o.ticket = 0u;
          *a.st = o;
        }
        if (observe) {
          hub.observe(phase(hub.node, cur));
          hub.close(a.n_steps);
        }
      }
    }
  }
  __syncthreads();
  if (*reinterpret_cast<volatile int *>(&s_ok) != 0) {
    if (live) {
      const long long gi = nd.node_off + row;
      if (sl.q == 0) {
        a.theta[gi] = th;
        a.theta_hat[gi] = thh;
        a.omega_hat[gi] = omh;
      }
      for (int s = sl.q; s < bsi; s += kSplitLPR)
        a.ring[nd.ring_off + ring_pos(s, row, Np)] = s_ring[(size_t)s * R + sl.rloc];
    }
    split_for_entries<kSplitLPR>(sloff, sllen, my_slices,
                                 [&](int at, int e) { a.sl_w[ebase + e] = s_w[at]; });
  }
  // no CTA may leave while a peer can still read its shared memory
  cluster.sync();
}

}  // namespace lev
