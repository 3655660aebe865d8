// lev_adj_grid.cuh -- grid-resident adjoint kernels for single networks whose
// CTAs all fit on the device at once.  Included once, from lev_engine.cu,
// after lev_grid.cuh and lev_adjoint.cuh.
//
// One cooperative launch runs a whole checkpoint segment:
//   adj_grid_fwd_kernel  the forward steps of the segment with the recording
//                        hooks of adj_fwd_kernel (pre-step theta_hat, post-step
//                        weights, per-step (g, r, sum cos, sum sin), r, theta),
//                        in the scheme of grid_kernel.  Bitwise the trajectory
//                        of adj_fwd_kernel and of the engine.
//   adj_grid_bwd_kernel  the reverse steps of the segment, last to first.  The
//                        adjoint node state (lam_theta, lam_theta_hat,
//                        lam_omega_hat, the omega gradient) stays in registers
//                        and lam_w in shared memory; the adjoint ring takes the
//                        red.add scatters in global memory.  lam_g(s) =
//                        lam_g(s+1) dg/dg + sum_i lam_th'_i dt S_i: every CTA
//                        publishes its part and every CTA adds the parts in the
//                        same order.
//   adj_grid_pair_kernel both at once, for the backward pass.
// All use the bounded waits of lev_grid.cuh (error flag on a timeout).

#pragma once

namespace lev {

// Edges per lane in flight together in the reverse steps, for kernels of at most
// `minb` CTAs per SM: four with 72 registers, six with 96.  T = 200, C = 50,
// accurate, backward us for four / six: N = 2,000, k = 16 (R = 64) 1,037 / 838;
// 5,000, k = 20 1,196 / 1,038; 10^4 (R = 128) 1,748 / 1,480.
__host__ __device__ constexpr int adj_bwd_unroll(int minb) { return minb == 2 ? 6 : 4; }

struct AdjGridFwdArgs {
  const NetDesc *net;  // adjoint copy: bsi = C + max_delay + 2
  NetState *st;
  const int *row_ptr;
  const long long *sl_off;
  const int *sl_len;
  const uint32_t *sl_cd;
  const float *w_in;   // SELL weights before the first step
  float *w_out;        // after the last step (may alias w_in)
  float *w_rec;        // weights after step k at w_rec + k*SL, or null
  float *theta;
  float *theta_hat;
  const float *omega;
  float *omega_hat;
  float *ring;
  const float *ring_src;  // ck_mode 1 and 3: the ring window of the initial state
  const float *drive;  // drive of step k at drive + k*N, or null
  const float *win;    // reservoir drive u_i = win_i * xin[k], or null
  const float *xin;
  float *thh_rec;      // theta_hat before step k at thh_rec + k*N, or null
  float4 *trace;       // (g, r, sum cos, sum sin) of step k at trace[k], or null
  float *r_out;        // r after step k at r_out[k], or null
  float *theta_out;    // theta after step k at theta_out + k*N, or null
  float2 *wsum;        // [4][8 * blocks] published sums, kNoSum at launch
  unsigned *bar;       // arrivals, zero at launch
  int *err;
  GridWait wait;  // bound of the barrier waits
  // the segment's checkpoint (theta, theta_hat, omega_hat, SELL weights, the
  // last max_delay+1 ring slots as [m][N], g): ck_mode 1 writes it from the
  // initial state (forward pass); 2 takes the initial state from it and
  // refills ring slots 0..max_delay, the unwrapped segment ring (backward
  // recompute); 3 writes it from the initial state and the ring window of
  // ring_src and goes on in the unwrapped ring `ring` (last segment of a forward
  // pass, which may be ring_src itself).  In 2 and 3 w0_out (if not null)
  // receives the initial weights
  int ck_mode;
  float *ck_theta, *ck_thh, *ck_omh, *ck_w, *ck_ring, *ck_g;
  float *w0_out;
  long long SL;
  int early;           // no delay is 0
  int sum_cap;         // sums staged per CTA (R < 256)
  int edge_cap;
  int n_steps;
  float dt;
};

// One segment's forward steps with the recording hooks, the scheme of
// grid_kernel (lev_grid.cuh): eight warps on R rows, a ninth exchanging sums
// and arrivals.  The body runs as CTA `cta` of a group of G CTAs (the whole
// grid, or one half of a paired launch).  Shared memory: sums float2 [sum_cap]
// (R < 256), sloff / sllen int [R/32], cd uint32 [edge_cap], w float [edge_cap].
template <int MATH, int R, int MINB>
__device__ __forceinline__ void adj_grid_fwd_body(const AdjGridFwdArgs &a, const int cta,
                                                  const unsigned G, unsigned char *smem) {
  constexpr int kUM = grid_walk_max(MATH, R, MINB);
  constexpr int LPR = 256 / R;
  constexpr int nslices = R / 32;
  constexpr bool kBlocks = R == 256;
  __shared__ float s_g;
  __shared__ int s_ok;
  __shared__ float2 s_part[8];

  const NetDesc nd = *a.net;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool exchange = warp == 8;
  const SplitLane sl = split_lane<LPR>(tid & 255);
  const int N = nd.N, bsi = nd.bsi, Np = nd.Np;
  const int row0 = cta * R;
  const int row = row0 + sl.rloc;
  const bool live = !exchange && row < N;
  const int nblocks = nd.ntiles;
  const int nsum = kBlocks ? nblocks : min(8 * nblocks, (int)G * nslices);

  float2 *s_sum = reinterpret_cast<float2 *>(smem);
  int *sloff = reinterpret_cast<int *>(s_sum + a.sum_cap);
  int *sllen = sloff + nslices;
  uint32_t *s_cd = reinterpret_cast<uint32_t *>(sllen + nslices);
  float *s_w = reinterpret_cast<float *>(s_cd + a.edge_cap);

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
  const bool restore = a.ck_mode == 2;
  const bool save = (a.ck_mode & 1) != 0;
  const bool unwrap = a.ck_mode >= 2;  // the segment runs in an unwrapped ring
  const float *w_src = restore ? a.ck_w : a.w_in;
  split_for_entries<LPR>(sloff, sllen, my_slices, [&](int at, int e) {
    s_cd[at] = a.sl_cd[ebase + e];
    const float w = w_src[ebase + e];
    s_w[at] = w;
    if (save) a.ck_w[ebase + e] = w;
    if (unwrap && a.w0_out) a.w0_out[ebase + e] = w;
  });
  const long long gi = nd.node_off + row;
  int deg = 0;
  float th = 0.0f, thh = 0.0f, om = 0.0f, omh = 0.0f;  // alike in the row's lanes
  if (live) {
    th = restore ? a.ck_theta[gi] : a.theta[gi];
    thh = restore ? a.ck_thh[gi] : a.theta_hat[gi];
    omh = restore ? a.ck_omh[gi] : a.omega_hat[gi];
    om = a.omega[gi];
    if (save && sl.q == 0) {
      a.ck_theta[gi] = th;
      a.ck_thh[gi] = thh;
      a.ck_omh[gi] = omh;
    }
    const int *rp = a.row_ptr + nd.rp_off + row;
    deg = rp[1] - rp[0];
  }
  NetState ns;
  if (restore) {
    // the state of a restored segment (adj_state_kernel mode 2)
    ns.g = a.ck_g[0];
    ns.r = 0.0f;
    ns.cur = nd.max_delay;
    ns.ticket = 0u;
    ns.t = 0;
    ns.rbuf = 0;
    ns.rpos = 0;
  } else {
    ns = *a.st;
  }
  float *ring = a.ring + nd.ring_off;
  if (save) {
    // ring window: theta(t - m) -> ck_ring[m][N], m = 0..max_delay
    const float *src = a.ring_src + nd.ring_off;
    if (live)
      for (int m = sl.q; m <= nd.max_delay; m += LPR) {
        int slot = ns.cur - m;
        slot += (slot < 0) ? bsi : 0;
        a.ck_ring[(long long)m * N + row] = src[(long long)slot * Np + row];
      }
    if (cta == 0 && tid == 0) a.ck_g[0] = ns.g;
  }
  int cur = unwrap ? nd.max_delay : ns.cur;
  float g = ns.g;
  const float dt = a.dt;
  __syncthreads();
  // unwrapped segment: theta(s0 - m) -> ring slot max_delay - m of every row
  // (from the checkpoint, so that the ring may be the one it was taken from),
  // read by every CTA's first gathers: all arrive once before step 0
  unsigned base = 0;
  if (unwrap) {
    if (live)
      for (int m = sl.q; m <= nd.max_delay; m += LPR)
        __stcg(ring + (long long)(nd.max_delay - m) * Np + row, a.ck_ring[(long long)m * N + row]);
    grid_arrive(a.bar);
    if (!grid_wait(a.bar, G, a.err, &s_ok, a.wait)) return;
    base = G;
  }

  if (!exchange) {
    const int len = sllen[sl.ws], eoff = sloff[sl.ws];
    for (int step = 0; step < a.n_steps; ++step) {
      if (step > 0 && !a.early) cta_barrier();
      // ---- predictor ----------------------------------------------------------
      if (a.thh_rec && live && sl.q == 0) a.thh_rec[(long long)step * N + gi] = thh;
      const float eps = sinf(wrap_pm_pi(th - thh));
      thh = thh + dt * omh;
      omh = omh + nd.kappa_w * dt * eps;
      // ---- edges ----------------------------------------------------------------
      const EdgeParams ep = {dt, nd.eta, nd.lam, __fmaf_rn(-nd.gamma, fabsf(eps), 1.0f),
                             nd.w_min, nd.w_max};
      auto gather = [&](uint32_t word) {
        const unsigned s0 = (unsigned)(cur - (int)(word & 255u));
        return __ldca(ring + (min(s0, s0 + (unsigned)bsi) * (unsigned)Np + (word >> 8)));
      };
      float local_sum;
      if (a.w_rec) {
        float *wr = a.w_rec + (long long)step * a.SL + ebase + eoff + sl.l;
        local_sum = split_walk<MATH, LPR, kUM>(s_cd + eoff, s_w + eoff, len, deg, sl, th, ep, gather,
                                          [&](int k, float w) { __stcs(wr + 32 * k, w); });
      } else {
        local_sum =
            split_walk<MATH, LPR, kUM>(s_cd + eoff, s_w + eoff, len, deg, sl, th, ep, gather);
      }
      if (step > 0) {
        cta_barrier();  // A
        if (*reinterpret_cast<volatile int *>(&s_ok) == 0) break;
        g = s_g;
      }
      // ---- integrate --------------------------------------------------------------
      int nxt = cur + 1;
      if (nxt == bsi) nxt = 0;
      float my_cos = 0.0f, my_sin = 0.0f;
      if (live) {
        float inc;
        if (a.drive || a.win) {
          float u = 0.0f;
          if (a.drive) u += a.drive[(long long)step * N + gi];
          if (a.win) u += a.win[gi] * a.xin[step];
          inc = dt * (om + g * local_sum - nd.alpha * eps + u);
        } else {
          inc = dt * (om + g * local_sum - nd.alpha * eps);
        }
        float x = th + inc;
        x = wrap_0_2pi(x);
        if (!isfinite(x)) x = 0.0f;
        th = x;
        if (sl.q == 0) {
          __stcg(ring + (size_t)nxt * Np + row, x);
          if (a.theta_out) a.theta_out[(long long)step * N + gi] = x;
        }
        lev_sincos<MATH>(x, &my_sin, &my_cos);
      }
      const float2 part = split_warp_sum<LPR>(my_cos, my_sin);
      if (lane == 0) s_part[warp] = part;
      cur = nxt;
      cta_barrier();  // B
    }
  } else {
    const float inv_N = 1.0f / (float)N;
    float r = ns.r;
    // r after `steps` steps and the gain of the next; false after a timeout
    auto close_step = [&](int steps) -> bool {
      float2 sums;
      if (!grid_sums<kBlocks>(a.wsum + ((steps - 1) & 3) * 8 * nblocks, nsum, nblocks, lane,
                              a.wait, s_sum, &sums))
        return false;
      r = order_parameter(sums.x, sums.y, inv_N);
      if (lane == 0 && cta == 0) {
        if (a.trace) a.trace[steps - 1] = make_float4(g, r, sums.x, sums.y);
        if (a.r_out) a.r_out[steps - 1] = r;
      }
      if (nd.ctrl) g = gain_controller(g, r, dt, nd);
      if (lane == 0) s_g = g;
      return true;
    };
    auto phases_of = [&](int steps) -> bool {
      const bool ok = lane != 0 || grid_poll(a.bar, base + (unsigned)steps * G, a.wait);
      return __all_sync(0xffffffffu, ok);
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
      if (step > 0) {
        if (!a.early) {
          ok = ok && phases_of(step);
          cta_barrier();
        }
        ok = ok && close_step(step);
        if (!ok) give_up();
        cta_barrier();  // A
        if (!ok) break;
        if (a.early) ok = phases_of(step);  // a timeout shows at the next barrier A
      }
      cur = (cur + 1 == bsi) ? 0 : cur + 1;
      cta_barrier();  // B
      grid_publish_part<R>(a.wsum, step, nblocks, nsum, cta, lane, s_part);
      __syncwarp();
      if (lane == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
    }
    if (!ok) give_up();
    if (ok && a.n_steps > 0 && cta == 0) {
      ok = close_step(a.n_steps);
      if (!ok) give_up();
      if (ok && lane == 0) {
        NetState o = ns;
        o.g = g;
        o.r = r;
        o.cur = cur;
        o.t = ns.t + a.n_steps;
        o.ticket = 0u;
        *a.st = o;
      }
    }
  }
  __syncthreads();
  if (*reinterpret_cast<volatile int *>(&s_ok) == 0) return;
  if (live && sl.q == 0) {
    a.theta[gi] = th;
    a.theta_hat[gi] = thh;
    a.omega_hat[gi] = omh;
  }
  split_for_entries<LPR>(sloff, sllen, my_slices,
                         [&](int at, int e) { a.w_out[ebase + e] = s_w[at]; });
}

struct AdjGridBwdArgs {
  const NetDesc *net;  // adjoint copy (ring_off: history ring, aux_off: adjoint ring)
  const int *row_ptr;
  const long long *sl_off;
  const int *sl_len;
  const uint32_t *sl_cd;
  const float *w_hist;   // weights before step seg_start + k at w_hist + k*SL
  const float *H;        // history ring: theta(tau) at slot tau - seg_start + max_delay
  const float *thh_hist; // theta_hat before step seg_start + k at thh_hist + k*N
  const float4 *trace;   // (g_s, r_{s+1}, sum cos, sum sin) of step seg_start + k at trace[k]
  const float *dLdr;     // dL/dr(s+1) at dLdr[s], or null
  const float *dLdth;    // dL/dtheta(s+1) at dLdth + s*N, or null
  float *grad_drive;     // at grad_drive + s*N, or null
  const float *win;      // reservoir drive (xin[s]); grad_win accumulated; or null
  const float *xin;
  float *grad_win;
  SplitArray lam_th;
  float *lam_thh;
  float *lam_omh;
  float *lam_w;          // SELL
  float *adj_ring;
  double *lam_g;         // [1]: in lam_g(seg_end), out lam_g(seg_start)
  float *grad_omega;     // accumulated
  double *lgp;           // [4][gpad] per-CTA lam_g parts, kNoPart at launch
  int gpad;
  unsigned *bar;         // two arrival counters, kGridBarPitch apart, zero at launch
  int *err;
  GridWait wait;  // bound of the barrier waits
  int early;             // no delay is 0: slot s+1 is complete one barrier earlier
  long long SL;
  long long seg_start;
  int n_steps;           // reverse steps seg_start + n_steps - 1 .. seg_start
  int edge_cap;
  float dt;
};

// A part of lam_g that has not been published yet: a NaN pattern that no
// published part has.
constexpr unsigned long long kNoPart = ~0ull;
__device__ __forceinline__ void st_relaxed_gpu(double *p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Barriers of the reverse body (cta_barrier is number 1).
__device__ __forceinline__ void cta_barrier_slot() {
  asm volatile("bar.sync 3, %0;" ::"n"(kGridThreads) : "memory");
}
__device__ __forceinline__ void cta_scatter_done() {  // edge warps: go on at once
  asm volatile("bar.arrive 2, %0;" ::"n"(kGridThreads) : "memory");
}
__device__ __forceinline__ void cta_scatter_wait() {
  asm volatile("bar.sync 2, %0;" ::"n"(kGridThreads) : "memory");
}

// Arrivals of the reverse steps: a CTA arrives for step k, its scatter done, on
// counter adj_arrival_counter(k); before it reads adjoint-ring slots in step k it
// waits until that counter holds adj_arrival_wait(k) arrivals per CTA, its
// own and every other's.  A total can only stand for "everyone" if nobody adds
// to it again before that wait.  With zero delays step k waits for step k-1 and
// arrives for k after the wait: one counter.  Without, step k waits for step k-2
// only, and a fast CTA's arrival for k-1 may come before a slow one's for k-2: the
// parts of lam_g, which let it go on, are published before the scatter.  So
// even and odd steps count apart.
__host__ __device__ constexpr int adj_arrival_counter(int k, int early) { return early ? k & 1 : 0; }
__host__ __device__ constexpr int adj_arrival_wait(int k, int early) { return early ? k >> 1 : k; }

// One segment's reverse steps.  Most of a step does not depend on the adjoint
// of the step reversed before: phases, weights, sines and cosines, the row's
// coupling sum S_i and the |eps| term.  All that comes first and is kept per
// entry in shared memory; what is left for after lam_g(s+1) is the node's
// lam_th', three multiply-adds and one scatter per edge.  And this step's part
// of lam_g, lam_th' dt S_i, is known before the scatter, so the exchange with
// the other CTAs runs while the scatter and the next step's first part do.
//
// Order of one reverse step k (s = seg_start + n_steps - 1 - k), edge warps | ninth warp:
//   edges, first part                | wait for everyone's arrival (scatter) of
//                                    | step k-2 (k-1 with zero delays)
//   ----------------- barrier D: adjoint slot s+1 is complete -------------------
//   read and clear slot s+1          | wait for the parts of step k-1; lam_g(s+1)
//   ----------------- barrier A: lam_g(s+1) -------------------------------------
//   lam_th', S_i parts               |
//   ----------------- barrier B: warp parts -------------------------------------
//   scatter; predictor               | publish this CTA's part, clear that of k-2
//   ----------------- scatter done (edge warps do not wait) ---------------------
//                                    | fence, arrive
// Slot s+1 takes scatters of the reverse steps s+1+d; without zero delays the
// last are those of step s+2, two reversed before.  Its clearing at step k is
// ordered by arrival k, which barrier D of step k+2 waits for, and the slot's
// next scatter comes from that step at the earliest (adj_slots).  Buffers of
// the parts as in grid_kernel.  Shared memory: sa float2 [edge_cap] (sin, w cos),
// cd uint32 [edge_cap], lw float [edge_cap] (lam_w; within a step c *
// lam_w(s+1)), sloff / sllen int [R/32].
//
// KEEP = false, for rows too long for 16 bytes per entry: no sa.  The edges are
// walked once, between A and B, scatter included; the exchange then waits for
// the walk, which is most of a step of such rows.  Backward us of 200 steps, per
// step launches / here: N = 30,000, k = 60 6,930 / 5,520; 15,000, k = 120 8,050 /
// 5,510; 9,000, k = 230 12,090 / 6,660; 4,000, k = 300 14,440 / 7,790.
template <int MATH, int R, int U, bool KEEP>
__device__ __forceinline__ void adj_grid_bwd_body(const AdjGridBwdArgs &a, const int cta,
                                                  const unsigned G, unsigned char *smem) {
  constexpr int LPR = 256 / R;
  constexpr int nslices = R / 32;
  __shared__ double s_red[8];
  __shared__ float s_lg;
  __shared__ int s_ok;

  const NetDesc nd = *a.net;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool exchange = warp == 8;
  const SplitLane sl = split_lane<LPR>(tid & 255);
  const unsigned mask = 0xffffffffu;
  const int N = nd.N, Np = nd.Np;
  const int row0 = cta * R;
  const int row = row0 + sl.rloc;
  const bool live = !exchange && row < N;
  const long long gi = nd.node_off + row;
  const int bsa = adj_slots(nd.max_delay);
  const float *H = a.H + nd.ring_off;
  float *AR = a.adj_ring + nd.aux_off;

  float2 *s_sa = reinterpret_cast<float2 *>(smem);
  uint32_t *s_cd = reinterpret_cast<uint32_t *>(s_sa + (KEEP ? a.edge_cap : 0));
  float *s_lw = reinterpret_cast<float *>(s_cd + a.edge_cap);
  int *sloff = reinterpret_cast<int *>(s_lw + a.edge_cap);
  int *sllen = sloff + nslices;

  const long long sl0 = nd.slice_base + row0 / 32;
  const int my_slices = max(0, min(nslices, (N - row0 + 31) / 32));
  const long long ebase = my_slices ? a.sl_off[sl0] : 0;
  for (int s = tid; s < nslices; s += blockDim.x) {
    sloff[s] = s < my_slices ? (int)(a.sl_off[sl0 + s] - ebase) : 0;
    sllen[s] = s < my_slices ? a.sl_len[sl0 + s] : 0;
  }
  if (tid == 0) s_ok = 1;
  __syncthreads();
  // entries in memory order within a slice: lane q of a row takes entries q,
  // q + LPR, ..., at 32k + ((l + q) mod 32) (one bank per lane)
  for (int s = 0; s < my_slices; ++s)
    for (int k = warp; k < sllen[s]; k += kGridThreads / 32) {
      const int at = sloff[s] + 32 * k + ((lane + (k & (LPR - 1))) & 31);
      s_cd[at] = a.sl_cd[ebase + sloff[s] + 32 * k + lane];
      s_lw[at] = a.lam_w[ebase + sloff[s] + 32 * k + lane];
    }
  int deg = 0;
  double lt = 0.0;  // lam_th; alike in the row's lanes
  float lthh = 0.0f, lomh = 0.0f, go = 0.0f;
  if (live) {
    lt = a.lam_th.get(gi).value();
    lthh = a.lam_thh[gi];
    lomh = a.lam_omh[gi];
    go = a.grad_omega[gi];
    const int *rp = a.row_ptr + nd.rp_off + row;
    deg = rp[1] - rp[0];
  }
  const float dt = a.dt;
  const float invN = 1.0f / (float)N;
  const float eta = nd.eta, gamma = nd.gamma, lam = nd.lam;
  const float w_min = nd.w_min, w_max = nd.w_max;
  const float decay = 1.0f - dt * lam;
  const int gpad = a.gpad;
  // derivatives of the gain controller at step s -> s+1
  auto controller = [&](const float4 &tr, float *dgdr, float *dgdg) {
    *dgdr = 0.0f;
    *dgdg = 1.0f;
    if (nd.ctrl) {
      const float g_s = tr.x, r1 = tr.y;
      const float pre = g_s + dt * (nd.beta * (nd.r0 - r1) - nd.mu * (g_s - nd.g_rest));
      const bool free = pre >= nd.g_min && pre <= nd.g_max;
      *dgdr = free ? -dt * nd.beta : 0.0f;
      *dgdg = free ? 1.0f - dt * nd.mu : 0.0f;
    }
  };
  __syncthreads();

  if (!exchange) {
    const int len = sllen[sl.ws], eoff = sloff[sl.ws];
    const int at0 = eoff + ((sl.l + sl.q) & 31);
    float th1 = 0.0f;  // theta(s+1): theta(s) of the step reversed before
    if (live) th1 = H[(long long)(a.n_steps + nd.max_delay) * Np + row];
    float lamg = (float)a.lam_g[0];  // lam_g(s+1)
    for (int k = 0; k < a.n_steps; ++k) {
      const long long s = a.seg_start + a.n_steps - 1 - k;
      const int kk = (int)(s - a.seg_start);
      const int hs = kk + nd.max_delay;  // history slot of theta(s)
      const int as_next = pos_mod(s + 1, bsa);
      const int as_s = pos_mod(s, bsa);
      // ---- first part: nothing here depends on the step reversed before --------
      const float4 tr = a.trace[kk];
      float th = 0.0f, thh = 0.0f;
      if (live) {
        th = H[(long long)hs * Np + row];
        thh = a.thh_hist[(long long)kk * N + gi];
      }
      const float diff = wrap_pm_pi(th - thh);
      const float eps = sinf(diff);
      float sn1, cs1;
      sincosf(th1, &sn1, &cs1);
      const EdgeParams ep = {dt, eta, lam, __fmaf_rn(-gamma, fabsf(eps), 1.0f), w_min, w_max};
      const float *w_s = a.w_hist + (long long)kk * a.SL + ebase + eoff + sl.l;
      float S_i = 0.0f, labs = 0.0f;
      // the row's entries: each(entry, word, c * lam_w(s+1), sin, w cos)
      auto walk = [&](auto each) {
        for (int kb = 0; kb < len; kb += LPR * U) {
          uint32_t p[U];
          float wv[U], dj[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int e = kb + LPR * u + sl.q;
            const bool in = e < deg;
            p[u] = in ? s_cd[at0 + 32 * e] : 0u;
            wv[u] = in ? __ldcs(w_s + 32 * e) : 0.0f;
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            dj[u] = (kb + LPR * u + sl.q < deg)
                        ? __ldg(H + ((unsigned)(hs - (int)(p[u] & 255u)) * (unsigned)Np + (p[u] >> 8))) - th
                        : 0.0f;
          float sn[U], cs[U];
          wrap_sincos_group<MATH>(dj, sn, cs);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int e = kb + LPR * u + sl.q;
            const float w = wv[u];
            S_i += w * sn[u];
            const float w_pre = edge_weight_free(ep, cs[u], w);
            const float lw = (e < deg) ? s_lw[at0 + 32 * e] : 0.0f;
            const float m = (w_pre >= w_min && w_pre <= w_max) ? lw : 0.0f;
            labs += m * cs[u];
            if (e < deg) each(e, p[u], m, sn[u], w * cs[u]);
          }
        }
#pragma unroll
        for (int off = 1; off < LPR; off *= 2) {
          S_i += __shfl_xor_sync(mask, S_i, off);
          labs += __shfl_xor_sync(mask, labs, off);
        }
      };
      if constexpr (KEEP)
        walk([&](int e, uint32_t, float m, float sn, float wcs) {
          s_lw[at0 + 32 * e] = m;
          s_sa[at0 + 32 * e] = make_float2(sn, wcs);
        });
      cta_barrier_slot();  // D
      float arv = 0.0f;
      if (live) arv = __ldcg(AR + (long long)as_next * Np + row);
      float extra = 0.0f;
      if (live && a.dLdth) extra = a.dLdth[s * N + gi];
      float dgdr, dgdg;
      controller(tr, &dgdr, &dgdg);
      const float dldr = a.dLdr ? a.dLdr[s] : 0.0f;
      if (k > 0) {
        cta_barrier();  // A
        if (*reinterpret_cast<volatile int *>(&s_ok) == 0) break;
        lamg = s_lg;
      }
      // ---- (A) adjoint of theta(s+1), complete; (B) integrate --------------------
      const float lam_r = dldr + lamg * dgdr;
      if (live) {
        const float Cm = tr.z * invN, Sm = tr.w * invN, r1 = tr.y;
        lt += arv;
        if (r1 > 0.0f) lt += lam_r * (Sm * cs1 - Cm * sn1) * invN / r1;
        if (a.dLdth) lt += extra;
      }
      const float lt1 = (float)lt;  // lam_th'
      float lsum = 0.0f;
      auto scatter = [&](int e, uint32_t p, float m, float sn, float wcs) {
        const float lam_S = lt1 * dt * tr.x;
        const float hq = dt * eta * ep.hebb;
        s_lw[at0 + 32 * e] = m * decay + lam_S * sn;
        const float lD = lam_S * wcs - m * hq * sn;
        const unsigned s0 = (unsigned)(as_s - (int)(p & 255u));
        atomicAdd(AR + (min(s0, s0 + (unsigned)bsa) * (unsigned)Np + (p >> 8)), lD);
        lsum -= lD;
      };
      if constexpr (!KEEP) walk(scatter);
      double part = sl.q == 0 ? (double)lt1 * dt * S_i : 0.0;
#pragma unroll
      for (int off = 16; off > 0; off /= 2) part += __shfl_down_sync(mask, part, off);
      if (lane == 0) s_red[warp] = part;
      cta_barrier();  // B
      // ---- scatter ------------------------------------------------------------------
      if constexpr (KEEP) {
#pragma unroll 4
        for (int e = sl.q; e < deg; e += LPR) {
          const float2 sa = s_sa[at0 + 32 * e];
          scatter(e, s_cd[at0 + 32 * e], s_lw[at0 + 32 * e], sa.x, sa.y);
        }
      }
#pragma unroll
      for (int off = 1; off < LPR; off *= 2) lsum += __shfl_xor_sync(mask, lsum, off);
      if (live) {
        go += lt1 * dt;
        if (sl.q == 0) {
          __stcg(AR + (long long)as_next * Np + row, 0.0f);
          if (a.grad_drive) a.grad_drive[s * N + gi] = lt1 * dt;
          if (a.grad_win) a.grad_win[gi] += lt1 * dt * a.xin[s];
        }
        // (D) predictor
        const float sgn = (eps > 0.0f) ? 1.0f : ((eps < 0.0f) ? -1.0f : 0.0f);
        const float leps = -lt1 * dt * nd.alpha - dt * eta * gamma * labs * sgn +
                           lomh * nd.kappa_w * dt;
        const float ldiff = leps * cosf(diff);
        lt += lsum + ldiff;
        const float lthh1 = lthh;
        lthh = lthh1 - ldiff;
        lomh = lomh + lthh1 * dt;
      }
      th1 = th;
      cta_scatter_done();
    }
  } else {
    double lamg = a.lam_g[0];
    float dgdg_prev = 1.0f;
    // lam_g(s+1) from lam_g(s+2) and the parts of reverse step `k`
    auto fold_parts = [&](int k) -> bool {
      const double *buf = a.lgp + (k & 3) * gpad;
      const unsigned long long t0 = global_ns();
      double sum = 0.0;
      constexpr int K = 4;
      for (int c0 = 0; c0 < (int)G; c0 += 32 * K) {
        unsigned long long v[K];
        for (;;) {
          bool ready = a.wait.extra == 0;
#pragma unroll
          for (int j = 0; j < K; ++j) {
            v[j] = 0ull;
            if (c0 + 32 * j + lane < (int)G)
              asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
                           : "=l"(v[j]) : "l"(buf + c0 + 32 * j + lane) : "memory");
            ready = ready && v[j] != kNoPart;
          }
          if (__all_sync(mask, ready)) break;
          if (__any_sync(mask, global_ns() - t0 > a.wait.ns)) return false;
        }
#pragma unroll
        for (int j = 0; j < K; ++j) sum += __longlong_as_double((long long)v[j]);
      }
#pragma unroll
      for (int off = 16; off > 0; off /= 2) sum += __shfl_down_sync(mask, sum, off);
      lamg = lamg * dgdg_prev + __shfl_sync(mask, sum, 0);
      if (lane == 0) s_lg = (float)lamg;
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
    for (int k = 0; k < a.n_steps; ++k) {
      const int kk = a.n_steps - 1 - k;
      const float4 tr = a.trace[kk];
      unsigned *bar = a.bar + kGridBarPitch * adj_arrival_counter(k, a.early);
      const unsigned arrived = (unsigned)adj_arrival_wait(k, a.early);
      if (ok && arrived > 0) {
        ok = lane != 0 || grid_poll(bar, arrived * G, a.wait);
        ok = __all_sync(mask, ok);
      }
      cta_barrier_slot();  // D
      if (k > 0) {
        ok = ok && fold_parts(k - 1);
        if (!ok) give_up();
        cta_barrier();  // A
        if (!ok) break;
      }
      float dgdr;
      controller(tr, &dgdr, &dgdg_prev);
      cta_barrier();  // B
      double part = lane < 8 ? s_red[lane] : 0.0;
#pragma unroll
      for (int off = 4; off > 0; off /= 2) part += __shfl_down_sync(mask, part, off);
      if (lane == 0) {
        unsigned long long v = (unsigned long long)__double_as_longlong(part);
        if (v == kNoPart) v = kNoPart >> 1;  // another NaN
        st_relaxed_gpu(a.lgp + (k & 3) * gpad + cta, v);
        st_relaxed_gpu(a.lgp + ((k + 2) & 3) * gpad + cta, kNoPart);
      }
      __syncwarp();
      cta_scatter_wait();
      if (lane == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    }
    if (!ok) give_up();
    if (ok && a.n_steps > 0 && cta == 0) {
      ok = fold_parts(a.n_steps - 1);
      if (!ok) give_up();
      if (ok && lane == 0) a.lam_g[0] = lamg;
    }
  }
  __syncthreads();
  if (*reinterpret_cast<volatile int *>(&s_ok) == 0) return;
  if (live && sl.q == 0) {
    a.lam_th.put(gi, SplitFloat::of(lt));
    a.lam_thh[gi] = lthh;
    a.lam_omh[gi] = lomh;
    a.grad_omega[gi] = go;
  }
  for (int s = 0; s < my_slices; ++s)
    for (int k = warp; k < sllen[s]; k += kGridThreads / 32)
      a.lam_w[ebase + sloff[s] + 32 * k + lane] =
          s_lw[sloff[s] + 32 * k + ((lane + (k & (LPR - 1))) & 31)];
}

template <int MATH, int R, int MINB>
__global__ void __launch_bounds__(kGridThreads, MINB) adj_grid_fwd_kernel(const AdjGridFwdArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  adj_grid_fwd_body<MATH, R, MINB>(a, blockIdx.x, gridDim.x, smem);
}

template <int MATH, int R, int MINB, bool KEEP>
__global__ void __launch_bounds__(kGridThreads, MINB) adj_grid_bwd_kernel(const AdjGridBwdArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  adj_grid_bwd_body<MATH, R, adj_bwd_unroll(MINB), KEEP>(a, blockIdx.x, gridDim.x, smem);
}

// Paired launch of the backward pass: CTAs [0, gf) recompute segment k-1
// into one record set while CTAs [gf, grid) reverse segment k from the
// other; each group has its own arrival counters and shares the SMs with the
// other, so the two latency-bound step chains overlap.  Every CTA of both
// groups is resident at once (cooperative launch).
template <int MATH, int R, int MINB>
__global__ void __launch_bounds__(kGridThreads, MINB)
    adj_grid_pair_kernel(const AdjGridFwdArgs f, const AdjGridBwdArgs b, const int gf) {
  extern __shared__ __align__(16) unsigned char smem[];
  if ((int)blockIdx.x < gf)
    adj_grid_fwd_body<MATH, R, MINB>(f, blockIdx.x, gf, smem);
  else
    adj_grid_bwd_body<MATH, R, adj_bwd_unroll(MINB), true>(b, blockIdx.x - gf, gridDim.x - gf, smem);
}

}  // namespace lev
