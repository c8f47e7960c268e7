// pimc_stage.cuh -- staging windows of one slot whose acceptance depends on
// the other paths (pair action), by a CTA.
//
// The windows of a slot follow one another: window n sees the accepted windows
// before it.  Walking them one by one (a warp, or a team of warps on one
// window) left most of a chain's time in the latency of single windows: 72 to
// 89 of 134 ms of a 512-chain physical sweep, 57 ms of one chain of 1024
// particles.  Here SLOT_B consecutive windows go together:
//  1. their proposals (bridge, potentials, links, mirror words) need only
//     their own paths, which no other window of the slot moves: a warp each;
//  2. a warp brackets each window's pair sums (scan_block) over the particles
//     outside the batch, which the batch does not move, and over the batch's
//     own paths twice, in place and as proposed: a lane per path;
//  3. one warp then decides the windows in order: the sums outside the batch,
//     plus for every earlier window of the batch the variant that its own
//     decision selects.  A window left open by its bracket is settled by the
//     whole CTA against the state at that point (accepted windows are written
//     as they are decided): from fixed-point positions, then from exact FP64
//     sums.
// So the decisions are those of the one-by-one walk, and the scans, all but a
// few percent of the work, run on every warp without barriers.
#pragma once
#include "pimc_kernels.cuh"

namespace pimc {

constexpr int SLOT_B = 32;

struct SlotScratch {
  float4 *pt;            // [SLOT_B][SLOT_B]: window i against path b: in place (sum, bound), as proposed
  double *x, *y, *vl;    // [SLOT_B][E]: beads, cached links of the proposals
  uint2 *cq;             // [SLOT_B][E]: mirror words, old and new
  uint2 *cf;             // [2 E]: one window's centres in fixed point
  unsigned *qn;          // [E]: one window's new words (exact sums)
  double *dw;            // [SLOT_B]: change of the action without pairs
  float *bt, *br, *lu;   // [SLOT_B]: sums outside the batch and their bound, log of the uniform
  int *m;                // [SLOT_B]
  float (*est)[2];       // [16]
  int *flag;             // [4]
  unsigned long long *q; // PQ_CAP neighbour queue per warp
  // E: beads of the longest window (ell + 1)
  static __host__ __device__ size_t bytes(int E, int nwarps) {
    const int e2 = (E + 1) & ~1;
    return sizeof(float4) * SLOT_B * SLOT_B + (size_t)SLOT_B * e2 * (3 * sizeof(double) + sizeof(uint2)) +
           sizeof(uint2) * 2 * e2 + sizeof(unsigned) * e2 + SLOT_B * (sizeof(double) + 4 * sizeof(int)) +
           16 * 8 + 16 + sizeof(unsigned long long) * PQ_CAP * (size_t)nwarps;
  }
  __device__ int carve(void *base, int E, int nwarps) {
    const int e2 = (E + 1) & ~1;
    unsigned char *p = (unsigned char *)base;
    auto take = [&](size_t n) { unsigned char *r = p; p += n; return r; };
    pt = (float4 *)take(sizeof(float4) * SLOT_B * SLOT_B);
    x = (double *)take(sizeof(double) * SLOT_B * e2);
    y = (double *)take(sizeof(double) * SLOT_B * e2);
    vl = (double *)take(sizeof(double) * SLOT_B * e2);
    dw = (double *)take(sizeof(double) * SLOT_B);
    q = (unsigned long long *)take(sizeof(unsigned long long) * PQ_CAP * nwarps);
    cq = (uint2 *)take(sizeof(uint2) * SLOT_B * e2);
    cf = (uint2 *)take(sizeof(uint2) * 2 * e2);
    qn = (unsigned *)take(sizeof(unsigned) * e2);
    bt = (float *)take(sizeof(float) * SLOT_B);
    br = (float *)take(sizeof(float) * SLOT_B);
    lu = (float *)take(sizeof(float) * SLOT_B);
    m = (int *)take(sizeof(int) * SLOT_B);
    est = (float(*)[2])take(16 * 8);
    flag = (int *)take(16);
    return e2;
  }
};

// one slot of a staging phase: windows from slice st over `len` slices, every
// particle in turn (pair action, no hard core or contact table, bounded
// decisions); the whole CTA calls it.  item0: the stream index of particle 0's
// window.  The tallies (attempts, accepts, beads) are thread 0's.
__device__ __forceinline__ void stage_slot(const CV &c, unsigned long long sweep, unsigned item0, int ell, int st,
                                  int len, void *scratch, double *red, int &n_att, int &n_acc,
                                  long long &n_bead) {
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M, dim = c.dim, lane = threadIdx.x & 31;
  const int warp = (int)(threadIdx.x >> 5), nwarps = (int)(blockDim.x >> 5);
  const double L = d.L, inv2L = d.inv2L, mhtau = -0.5 * d.tau;
  const float gh = (float)(-d.mhtau_g);
  SlotScratch S;
  const int E = S.carve(scratch, min(ell, len) + 1, nwarps);
  auto slc = [&](int t) { return st + t < M ? st + t : st + t - M; };
  for (int n0 = 0; n0 < N; n0 += SLOT_B) {
    const int nb = min(SLOT_B, N - n0);
    // window lengths and Metropolis uniforms, a lane per window
    if (warp == 0 && lane < nb) {
      const Stream ss = make_stream(d, sweep, PH_STAGE, item0 + n0 + lane);
      S.m[lane] = min(len, 2 + (int)(ss.uni(DRAW_CHOICE) * (ell - 1)));
      const double u = ss.uni(DRAW_ACCEPT);
      S.lu[lane] = u > 0.0 ? logf((float)u) : -INFINITY;
    }
    __syncthreads();
    // 1. proposals
    for (int i = warp; i < nb; i += nwarps) {
      const int n = n0 + i, nx = c.next[n], m = S.m[i];
      if (!check_ok(m >= 2 && m <= WMAX && m < E && m < M, DERR_WINDOW, d)) continue;
      const bool wr = st + m >= M;
      const int oe = wr ? nx : n, je = slc(m);
      const GenDraws dr = gen_draws(make_stream(d, sweep, PH_STAGE, item0 + n));
      double *X = S.x + (size_t)i * E, *Y = S.y + (size_t)i * E, *V = S.vl + (size_t)i * E;
      uint2 *cq = S.cq + (size_t)i * E;
      const double sx = c.X(0, n, st), sy = c.Xd(1, n, st);
      double ex = c.X(0, oe, je), ey = c.Xd(1, oe, je);
      if (abs_gt(sx - ex, L)) unwrap_end(sx, ex, L);
      if (dim > 1 && abs_gt(sy - ey, L)) unwrap_end(sy, ey, L);
      bridge_beads(c, m, dr, sx, sy, ex, ey, X, Y, lane);
      __syncwarp();
      double dw = 0.0, vlast = 0.0;
      // links behind the bead: lane t of a chunk forms link t - 1 -> t; the chunk's
      // first takes the bead before from the last lane
      for (int t0 = 0; t0 <= m; t0 += 32) {
        const int t = t0 + lane;
        double v = 0.0;
        if (t <= m) {
          double qx = t == 0 ? sx : (t == m ? ex : X[t]), qy = t == 0 ? sy : (t == m ? ey : Y[t]);
          qx = teleport_s<true>(qx, L, inv2L);
          qy = dim > 1 ? teleport_s<true>(qy, L, inv2L) : 0.0;
          X[t] = qx;
          Y[t] = qy;
          v = vext(d, qx, qy);
          const int a = st + t;
          cq[t] = make_uint2(a < M ? c.Q(n, a) : c.Q(nx, a - M), qpos(d, qx, qy));
        }
        double vp = __shfl_up_sync(0xffffffffu, v, 1);
        if (lane == 0) vp = vlast;
        vlast = __shfl_sync(0xffffffffu, v, 31);
        if (t >= 1 && t <= m) {
          const double link = mhtau * (vp + v);
          const int a = st + t - 1;
          V[t - 1] = link;
          dw += link - (a < M ? c.Vl(n, a) : c.Vl(nx, a - M));
        }
      }
      dw = warp_sum(dw);
      if (lane == 0) S.dw[i] = dw;
    }
    __syncthreads();
    // 2. brackets of the pair sums
    for (int i = warp; i < nb; i += nwarps) {
      const int n = n0 + i, m = S.m[i];
      const unsigned *cq = reinterpret_cast<const unsigned *>(S.cq + (size_t)i * E);
      const ScanSkip<2> skip{n, -1, true};
      PairEst e = {0.f, 0.f, 0.f, 0.f, 0, 0};
      scan_mirror<2>(c, st, m, cq, skip, 0, 1, e, lane, NoStop(), n0);
      scan_bounds(d, e);
      float t, r, tb, rb;
      est_lane(e, -1.f, t, r);
      // the batch's paths: in place, and for earlier windows as proposed
      const int b = n0 + lane, bl = min(b, N - 1), ib = bl - n0;
      const bool wraps = st + m >= M;
      const int nxb = wraps ? c.next[bl] : bl;
      auto word = [&](int q) { return st + q < M ? c.Q(bl, st + q) : c.Q(nxb, st + q - M); };
      PairEst o = {0.f, 0.f, 0.f, 0.f, 0, 0}, p = {0.f, 0.f, 0.f, 0.f, 0, 0};
      scan_block<2>(d, m, cq, word, [&](int) { return b < N && b != n; }, o);
      scan_bounds(d, o);
      est_lane(o, -1.f, tb, rb);
      if (lane > i) {  // a later window's path stays in place
        t += tb;
        r += rb;
      }
      t = warp_sum(t);
      r = warp_sum(r);
      if (lane == 0) {
        S.bt[i] = t;
        S.br[i] = r;
      }
      float4 w = make_float4(tb, rb, 0.f, 0.f);
      if (i > 0) {
        const int mb = S.m[ib];
        const uint2 *cb = S.cq + (size_t)ib * E;
        scan_block<2>(d, m, cq, [&](int q) { return q >= 1 && q < mb ? cb[q].y : word(q); },
                      [&](int) { return lane < i; }, p);
        scan_bounds(d, p);
        est_lane(p, -1.f, w.z, w.w);
      }
      S.pt[i * SLOT_B + lane] = w;
    }
    __syncthreads();
    // 3. decisions in order
    unsigned acc = 0u;  // accepted windows of the batch (warp 0)
    auto write = [&](int i) {  // window i's beads and links, by warp 0
      const int n = n0 + i, nx = c.next[n], m = S.m[i];
      const double *X = S.x + (size_t)i * E, *Y = S.y + (size_t)i * E, *V = S.vl + (size_t)i * E;
      const uint2 *cq = S.cq + (size_t)i * E;
      for (int t = lane; t < m; t += 32) {
        const int a = st + t, o = a < M ? n : nx, j = a < M ? a : a - M;
        if (t > 0) {
          c.X(0, o, j) = X[t];
          if (dim > 1) c.X(1, o, j) = Y[t];
          c.xq[(size_t)j * c.ldn + o] = cq[t].y;
        }
        c.Vl(o, j) = V[t];
      }
    };
    int i = 0;
    while (true) {
      if (warp == 0) {
        for (; i < nb; ++i) {
          const float4 w = S.pt[i * SLOT_B + lane];
          const bool on = lane < i, moved = (acc >> lane) & 1u;
          const float t = S.bt[i] + warp_sum(on ? (moved ? w.z : w.x) : 0.f);
          const float r = S.br[i] + warp_sum(on ? (moved ? w.w : w.y) : 0.f);
          const float dw = (float)S.dw[i];
          const int dec = decide_f(fmaf(gh, t, dw), fabsf(gh) * r + 1e-6f * fabsf(dw), S.lu[i]);
          if (dec == -1) break;
          if (dec == 1) {
            acc |= 1u << i;
            write(i);
          }
        }
        if (lane == 0) S.flag[0] = i;
      }
      __syncthreads();
      i = S.flag[0];
      if (i >= nb) break;
      // window i stayed open: fixed point, then exact sums, by the whole CTA
      const int n = n0 + i, nx = c.next[n], m = S.m[i];
      const double *X = S.x + (size_t)i * E, *Y = S.y + (size_t)i * E;
      for (int k = threadIdx.x; k <= m; k += blockDim.x) {
        const int a = st + k, o = a < M ? n : nx, j = a < M ? a : a - M;
        S.cf[2 * k] = make_uint2(fix32(d, c.X(0, o, j)), fix32(d, c.Xd(1, o, j)));
        S.cf[2 * k + 1] = make_uint2(fix32(d, X[k]), fix32(d, Y[k]));
        S.qn[k] = S.cq[(size_t)i * E + k].y;
      }
      __syncthreads();
      PairEst e = {0.f, 0.f, 0.f, 0.f, 0, 0};
      scan_fixed<2>(c, st, m, S.cf, ScanSkip<2>{n, -1, true}, warp, nwarps, e, lane);
      float t, r;
      est_lane(e, -1.f, t, r);
      t = warp_sum(t);
      r = warp_sum(r);
      if (lane == 0) {
        S.est[warp][0] = t;
        S.est[warp][1] = r;
      }
      __syncthreads();
      t = r = 0.f;
      for (int w = 0; w < nwarps; ++w) {
        t += S.est[w][0];
        r += S.est[w][1];
      }
      const float dw = (float)S.dw[i];
      int dec = decide_f(fmaf(gh, t, dw), fabsf(gh) * r + 1e-6f * fabsf(dw), S.lu[i]);
      if (dec == -1) {
        const WindowSeg seg{&c, n, nx, st, M, X, Y, S.qn};
        const int per = (m + nwarps - 1) / nwarps, t0 = min(m, warp * per), t1 = min(m, t0 + per);
        double w2[2] = {0.0, 0.0};
        if (t0 < t1) segment_pairs(c, seg, t0, t1, true, true, S.q + (size_t)warp * PQ_CAP, w2[0], w2[1], lane);
        block_sum_k<2>(w2, red);
        GenDraws dr = gen_draws(make_stream(d, sweep, PH_STAGE, item0 + n));
        dec = metropolis(d, S.dw[i] + (w2[1] - w2[0]), dr);
      }
      if (warp == 0 && dec) {
        acc |= 1u << i;
        write(i);
      }
      ++i;
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      n_att += nb;
      n_acc += __popc(acc);
      for (int k = 0; k < nb; ++k) n_bead += S.m[k] - 1;
    }
    __syncthreads();
  }
}

// the same out of line with the view by value, for the fused sweep kernel,
// whose other phases would lose registers to it (4 % of a batch of small
// pair-free chains)
static __device__ __noinline__ void stage_slot_call(CV c, unsigned long long sweep, unsigned item0, int ell, int st,
                                                    int len, void *scratch, double *red, int &n_att, int &n_acc,
                                                    long long &n_bead) {
  stage_slot(c, sweep, item0, ell, st, len, scratch, red, n_att, n_acc, n_bead);
}

}  // namespace pimc
