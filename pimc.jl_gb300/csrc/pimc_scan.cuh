// pimc_scan.cuh -- bounded estimates of a move's pair sums, every particle of
// the moved slices scanned, for windows of at most WMAX links.
//
// A move's pair sums only decide its Metropolis test, so a sweep brackets them
// in FP32 and evaluates them in FP64 only when the bracket straddles the
// threshold.  Two brackets: from the 16-bit mirror (integers and FP32 alone,
// within about half a percent of the sums), then, for the few moves that it
// leaves open, from the positions in 32-bit fixed point (two FP64
// instructions per bead, within about 1e-5).
//
// A lane follows one particle's path through the window's slices (past slice M
// its successor), so a pair's exponential at a slice serves both links that
// meet there, the words of a slice are read once for every centre (the old
// and the new bead of each moving path), and "not the moving path itself" is a
// test of the lane's particle alone.  Scanning link by link instead read each
// row twice and formed each exponential twice, per centre: 2.3 times the
// instructions, which bound this scan (one warp issues every 5 cycles or so).
#pragma once

namespace pimc {

__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// the centres of a scan: NC = 2, one moving path (old, new bead); NC = 4, two
// (old 1, new 1, old 2, new 2).  Centre k of path p leaves out p itself and,
// when both(k), the other moving path.
template <int NC>
struct ScanSkip {
  int p1, p2;      // the moving paths' particles at the window's start (p2 -1: one path)
  bool old_both;   // the old beads leave the other moving path out as well
  __device__ __forceinline__ bool operator()(int k, int b) const {
    if (NC == 2) return b == p1;
    const int own = k < 2 ? p1 : p2;
    return b == own || ((k & 1) || old_both ? (b == p1 || b == p2) : false);
  }
};

// a lane's sums over one particle, from the mirror, added to e: old and new
// sums of exp(-r_a^2/2s^2) + exp(-r_b^2/2s^2) over the links whose start surely
// has the particle within reach (PairEst so, sn) and over those where it may
// (bo, bn: scan_bounds turns both into a sum and a bound).  cq[t * NC + k]:
// mirror word of centre k at bead t, t = 0 .. m; word(t): the particle's; on(k):
// whether centre k counts it.  Sixteen instructions per bead and centre bound
// the scan: coordinates as the upper halves of words, so that a difference
// wraps by itself and converts exactly.
template <int NC, class Word, class On>
__device__ __forceinline__ void scan_block(const ChainDesc &d, int m, const unsigned *cq, const Word &word,
                                           const On &on, PairEst &e) {
  const float cx = d.est_x;
  float lo[NC], hi[NC], ep[NC], wi[NC], wm[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    lo[k] = on(k) ? d.est_lo : -1.f;
    hi[k] = on(k) ? d.est_hi : -1.f;
    ep[k] = wi[k] = wm[k] = 0.f;
  }
  // the slices' words four beads ahead: a step takes a few hundred cycles, a
  // word from L2 up to a thousand
  unsigned q0 = word(0), q1 = word(min(1, m)), q2 = word(min(2, m)), q3 = word(min(3, m));
  for (int t = 0; t <= m; ++t) {
    const unsigned qx = q0 << 16, qy = q0 & 0xffff0000u;
    q0 = q1;
    q1 = q2;
    q2 = q3;
    if (t + 4 <= m) q3 = word(t + 4);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const unsigned w = cq[t * NC + k];
      const float dx = (float)(int)((w << 16) - qx), dy = (float)(int)((w & 0xffff0000u) - qy);
      const float f = fmaf(dx, dx, dy * dy), x = ex2_approx(f * cx), v = ep[k] + x;
      if (k & 1) {
        e.sn = fmaf(wi[k], v, e.sn);
        e.bn = fmaf(wm[k], v, e.bn);
      } else {
        e.so = fmaf(wi[k], v, e.so);
        e.bo = fmaf(wm[k], v, e.bo);
      }
      ep[k] = x;
      wi[k] = f < lo[k] ? 1.f : 0.f;
      wm[k] = f < hi[k] ? 1.f : 0.f;
    }
  }
  e.ko += m * (NC / 2);
  e.kn += m * (NC / 2);
}

// the lane's sums [sure, may] of scan_block as the middle of the interval that
// holds the exact sum, and its half width.  An end within reach is off by at
// most est_eps of its value; one beyond by at most est_eps times est_far (the
// error bound grows with d^2, but x d^2 falls past the reach), once per link
// (ko, kn).
__device__ __forceinline__ void scan_bounds(const ChainDesc &d, PairEst &e) {
  const float far = d.est_eps * d.est_far;
  const float mo = 0.5f * (e.so + e.bo), mn = 0.5f * (e.sn + e.bn);
  e.bo = 0.5f * (e.bo - e.so) + d.est_eps * e.bo + far * (float)e.ko;
  e.bn = 0.5f * (e.bn - e.sn) + d.est_eps * e.bn + far * (float)e.kn;
  e.so = mo;
  e.sn = mn;
}

// the lane's sums over the particles 32 (part, part + nparts, ...) + lane, the
// block `leave` left out; stop(e) ends the scan early and is asked after every
// block of particles
template <int NC, class Stop>
__device__ __forceinline__ bool scan_mirror(const CV &c, int j0, int m, const unsigned *cq,
                                            const ScanSkip<NC> &skip, int part, int nparts, PairEst &e,
                                            int lane, const Stop &stop, int leave = -1) {
  const int N = c.N, M = c.M;
  const bool wraps = j0 + m >= M;
  for (int b0 = 32 * part; b0 < N; b0 += 32 * nparts) {
    if (b0 == leave) continue;
    const int b = b0 + lane, bl = min(b, N - 1);
    const int nb = wraps ? c.next[bl] : bl;
    scan_block<NC>(*c.d, m, cq, [&](int t) { return j0 + t < M ? c.Q(bl, j0 + t) : c.Q(nb, j0 + t - M); },
                   [&](int k) { return b < N && !skip(k, b); }, e);
    if (stop(e)) return true;
  }
  return false;
}
// (stop sees the raw sums; the caller applies scan_bounds)

// 32-bit fixed point of a coordinate on the periodic box (a wrapped difference
// is the minimum image), one FP64 instruction
__device__ __forceinline__ unsigned fix32(const ChainDesc &d, double x) {
  return (unsigned)__double2loint(fma(x, d.f_scale, 6755399441055744.0));
}

// exact a + b = s + err (Knuth's TwoSum), for sums over blocks
__device__ __forceinline__ void two_sum(float &s, float &lo, float v) {
  const float t = s + v, z = t - s;
  lo += (s - (t - z)) + (v - z);
  s = t;
}

// the same sums from the positions in fixed point; cf[t * NC + k]: centre k at
// bead t.  A coordinate is within half a unit of the exact one (2L / 2^32),
// the rest is FP32 rounding: relative 8e-7 (1 + y) plus est2 per exponential
template <int NC>
__device__ __forceinline__ void scan_fixed(const CV &c, int j0, int m, const uint2 *cf,
                                           const ScanSkip<NC> &skip, int part, int nparts, PairEst &e,
                                           int lane) {
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M;
  const bool wraps = j0 + m >= M;
  const float u = d.f_unit, rc2 = d.rc2_s;
  const float r_lo = rc2 * (1.f - 2e-6f) - 8.f * u * d.rc_s, r_hi = rc2 * (1.f + 2e-6f) + 8.f * u * d.rc_s;
  const float cy = d.inv2s2_s;
  float lo_s[2] = {0.f, 0.f};
  for (int b0 = 32 * part; b0 < N; b0 += 32 * nparts) {
    const int b = b0 + lane, bl = min(b, N - 1);
    const int nb = wraps ? c.next[bl] : bl;
    bool on[NC];
#pragma unroll
    for (int k = 0; k < NC; ++k) on[k] = b < N && !skip(k, b);
    float ep[NC], rp[NC], wp[NC], gp[NC], sb[2] = {0.f, 0.f};
#pragma unroll
    for (int k = 0; k < NC; ++k) ep[k] = rp[k] = wp[k] = gp[k] = 0.f;
    for (int t = 0; t <= m; ++t) {
      const int a = j0 + t, j = a < M ? a : a - M, n = a < M ? bl : nb;
      const unsigned qx = fix32(d, c.X(0, n, j)), qy = fix32(d, c.Xd(1, n, j));
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const uint2 ct = cf[t * NC + k];
        const float dx = (float)(int)(ct.x - qx) * u, dy = (float)(int)(ct.y - qy) * u;
        const float r2 = fmaf(dx, dx, dy * dy), y = r2 * cy;
        const float x = ex2_approx(y * -1.44269504f);
        const float r = fmaf(x, fmaf(8e-7f, y, d.est2), 1e-30f);
        const float v = ep[k] + x, ve = rp[k] + r;
        float &bd = (k & 1) ? e.bn : e.bo;
        sb[k & 1] = fmaf(wp[k], v, sb[k & 1]);
        bd = fmaf(wp[k], ve, bd);
        bd = fmaf(gp[k], v + ve, bd);
        ep[k] = x;
        rp[k] = r;
        const bool in = on[k] && r2 < r_lo, may = on[k] && r2 <= r_hi;
        gp[k] = may && !in ? 0.5f : 0.f;
        wp[k] = in ? 1.f : gp[k];
      }
    }
    // a block's FP32 sum: at most m NC / 2 terms (the bound below); blocks add
    // exactly
    e.bo += 1.5e-7f * (float)(m * (NC / 2) + 1) * sb[0];
    e.bn += 1.5e-7f * (float)(m * (NC / 2) + 1) * sb[1];
    two_sum(e.so, lo_s[0], sb[0]);
    two_sum(e.sn, lo_s[1], sb[1]);
  }
  e.so += lo_s[0];
  e.sn += lo_s[1];
  e.ko += 2;
  e.kn += 2;
  // the bounds' own additions
  e.bo *= 1.001f;
  e.bn *= 1.001f;
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// one contact term log(1 + T(|d1|, |d2|) / rel0) in FP32 from fixed-point
// differences (a1x, a1y) at a slice and (a2x, a2y) at the next: its value and a
// bound on the distance from contact_lnU; a negative bound: not settled here
// (where 1 + T / rel0 is small), the FP64 form decides.  T's weights are off by
// the radii's rounding (5e-7 and three units), bounded with the cell's slopes
// (next to a kink of the bilinear table the neighbouring cells' too); rel0's
// exponent by its own.  Lanes that do not count (act) read the first cell.
__device__ __forceinline__ float2 contact_term(const ChainDesc &d, bool act, int a1x, int a1y, int a2x, int a2y) {
  const float u = d.f_unit;
  const float x1 = (float)a1x * u, y1 = (float)a1y * u, x2 = (float)a2x * u, y2 = (float)a2y * u;
  const float r[2] = {sqrt_approx(fmaf(x1, x1, y1 * y1)), sqrt_approx(fmaf(x2, x2, y2 * y2))};
  int cell[2];
  float w[2], dp[2];
  bool kink = false;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float p = r[q] * d.ct_invh, last = (float)(d.ct_n - 1), f = fminf(floorf(p), last - 1.f);
    const bool past = p * (1.f - 8e-7f) - 3.f * u * d.ct_invh > last;  // clamped
    dp[q] = past ? 0.f : p * 8e-7f + 3.f * u * d.ct_invh;
    cell[q] = (int)f;
    w[q] = past ? 1.f : p - f;
    kink = kink || (!past && ((w[q] < dp[q] && f > 0.f) || w[q] > 1.f - dp[q]));
  }
  const size_t at = act ? (size_t)cell[0] * (d.ct_n - 1) + cell[1] : 0;
  const float4 g = __ldg(d.ct_cells + at);  // T at (i, j), (i, j+1), (i+1, j), (i+1, j+1)
  const float s0 = fmaf(w[1], g.y - g.x, g.x), s1 = fmaf(w[1], g.w - g.z, g.z), T = fmaf(w[0], s1 - s0, s0);
  const float big = fmaxf(fmaxf(fabsf(g.x), fabsf(g.y)), fmaxf(fabsf(g.z), fabsf(g.w)));
  float gx = fmaxf(fabsf(g.z - g.x), fabsf(g.w - g.y)), gy = fmaxf(fabsf(g.y - g.x), fabsf(g.w - g.z));
  if (act && kink)
    for (int i = max(cell[0] - 1, 0); i <= min(cell[0] + 1, d.ct_n - 2); ++i)
      for (int j = max(cell[1] - 1, 0); j <= min(cell[1] + 1, d.ct_n - 2); ++j) {
        const float4 h = __ldg(d.ct_cells + (size_t)i * (d.ct_n - 1) + j);
        gx = fmaxf(gx, fmaxf(fabsf(h.z - h.x), fabsf(h.w - h.y)));
        gy = fmaxf(gy, fmaxf(fabsf(h.y - h.x), fabsf(h.w - h.z)));
      }
  const float dT = 2.f * (dp[0] * gx + dp[1] * gy) + 8e-7f * big;
  // the physical rules take the signed difference of the two separations, the
  // reference its components' absolute values
  const bool phys = (d.flags & PF_PHYS) != 0;
  const int ix = phys ? (int)((unsigned)a1x - (unsigned)a2x) : abs(a1x) - abs(a2x);
  const int iy = phys ? (int)((unsigned)a1y - (unsigned)a2y) : abs(a1y) - abs(a2y);
  const float ex = (float)ix * u, ey = (float)iy * u;
  const float z = fmaf(ex, ex, ey * ey) * d.ct_c4;  // log2 of exp(dd / 4 tau)
  const float dz = z * 8e-7f + 8.f * u * (fabsf(ex) + fabsf(ey) + u) * d.ct_c4;
  const float K = ex2_approx(z) * d.ct_4pt, q = T * K, p1 = 1.f + q;
  const float dq = dT * K * 1.00001f + fabsf(q) * (dz + 6e-7f);
  // lg2.approx: within 2^-22 (about p1 = 1) or two ulp
  const float v = __logf(p1), dv = __fdividef(1.31f * dq, p1) + 4e-7f * (1.f + fabsf(v));
  const bool settled = z < 100.f && p1 > 1e-4f && dq < 0.2f * p1 && dv < 2e-3f;
  return make_float2(v, settled ? dv : -1.f);
}

// the contact chains' bracket: per link the table's pair action itself over the
// partners within reach at the link's start, from the positions in fixed
// point; cur(k, t, x, y): centre k's position at bead t (terms settled in
// FP64); ring: RING_C words of the warp.  The exact sums spend some 150 FP64
// instructions a term.  Here the lanes test a term for weight -- past ct_neg at
// both ends and with a small exponent it is below 1e-7, three of four terms
// within reach of a dense cloud -- and queue the others, evaluated 32 at a time.
constexpr int RING_C = 64;  // at most 31 + 32 in use
template <int NC, class Cur>
__device__ __forceinline__ void scan_contact(const CV &c, int j0, int m, const uint2 *cf,
                                             const ScanSkip<NC> &skip, int part, int nparts, PairEst &e,
                                             int lane, unsigned *ring, const Cur &cur) {
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M;
  const bool wraps = j0 + m >= M;
  const float u = d.f_unit, rc2 = d.rc2_s, neg2 = d.ct_neg * d.ct_neg;
  const float r_lo = rc2 * (1.f - 2e-6f) - 8.f * u * d.rc_s, r_hi = rc2 * (1.f + 2e-6f) + 8.f * u * d.rc_s;
  const unsigned lt = (1u << lane) - 1u;
  int head = 0, tail = 0;
  float sa = 0.f, na = 0.f, lo_o = 0.f, lo_n = 0.f;  // sum of magnitudes, terms left out
  auto flush = [&](int cnt) {
    if (lane < cnt) {
      const unsigned w = ring[(head + lane) & (RING_C - 1)];
      const int b = (int)(w & 0x1fffu), t = (int)((w >> 13) & 0x7fu), k = (int)((w >> 20) & 3u);
      const float wt = (w >> 22) & 1u ? 0.5f : 1.f;
      const int ap = j0 + t - 1, at = j0 + t;
      const int nb = wraps ? c.next[b] : b;
      const int jp = ap < M ? ap : ap - M, np = ap < M ? b : nb, j = at < M ? at : at - M, n = at < M ? b : nb;
      const double px = c.X(0, np, jp), py = c.Xd(1, np, jp), qx = c.X(0, n, j), qy = c.Xd(1, n, j);
      const uint2 cp = cf[(t - 1) * NC + k], ct = cf[t * NC + k];
      float2 v = contact_term(d, true, (int)(cp.x - fix32(d, px)), (int)(cp.y - fix32(d, py)),
                              (int)(ct.x - fix32(d, qx)), (int)(ct.y - fix32(d, qy)));
      if (v.y < 0.f) {
        double ax, ay, nx, ny;
        cur(k, t - 1, ax, ay);
        cur(k, t, nx, ny);
        v.x = (float)contact_link(d, ax, ay, px, py, nx, ny, qx, qy);
        v.y = 1e-7f * fabsf(v.x);
      }
      if (k & 1) two_sum(e.sn, lo_n, wt * v.x);
      else two_sum(e.so, lo_o, wt * v.x);
      sa += fabsf(v.x);
      e.bo += v.y + (1.f - wt) * fabsf(v.x);
    }
    head += cnt;
    __syncwarp();
  };
  for (int b0 = 32 * part; b0 < N; b0 += 32 * nparts) {
    const int b = b0 + lane, bl = min(b, N - 1);
    const int nb = wraps ? c.next[bl] : bl;
    int px[NC], py[NC];
    float wp[NC], rp[NC];  // reach at the slice before (1, 0.5 unsettled, 0), its r^2
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      px[k] = py[k] = 0;
      wp[k] = rp[k] = 0.f;
    }
    double xn = c.X(0, bl, j0), yn = c.Xd(1, bl, j0);
    for (int t = 0; t <= m; ++t) {
      const unsigned qx = fix32(d, xn), qy = fix32(d, yn);
      if (t < m) {  // the next slice's position
        const int a = j0 + t + 1, j = a < M ? a : a - M, n = a < M ? bl : nb;
        xn = c.X(0, n, j);
        yn = c.Xd(1, n, j);
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const uint2 ct = cf[t * NC + k];
        const int ix = (int)(ct.x - qx), iy = (int)(ct.y - qy);
        const float dx = (float)ix * u, dy = (float)iy * u, r2 = fmaf(dx, dx, dy * dy);
        if (t > 0) {
          // an upper bound of dd (either rule): the components' signed difference
          const float ex = dx - (float)px[k] * u, ey = dy - (float)py[k] * u;
          const bool light = fminf(rp[k], r2) > neg2 && fmaf(ex, ex, ey * ey) * d.ct_c4 < 6.6f;
          const bool on = wp[k] != 0.f;
          if (on && light) na += 1.f;
          const bool push = on && !light;
          const unsigned mk = __ballot_sync(0xffffffffu, push);
          if (push)
            ring[(tail + __popc(mk & lt)) & (RING_C - 1)] =
                (unsigned)b | ((unsigned)t << 13) | ((unsigned)k << 20) | (wp[k] != 1.f ? 1u << 22 : 0u);
          tail += __popc(mk);
          __syncwarp();
          if (tail - head >= 32) flush(32);
        }
        const bool cnt = b < N && !skip(k, b);
        wp[k] = cnt && r2 < r_lo ? 1.f : (cnt && r2 <= r_hi ? 0.5f : 0.f);
        rp[k] = r2;
        px[k] = ix;
        py[k] = iy;
      }
    }
  }
  if (tail > head) flush(tail - head);
  e.so += lo_o;
  e.sn += lo_n;
  e.ko += 2;
  e.kn += 2;
  // the light terms, and for terms of either sign what est_lane and the sums
  // over the warps need of the magnitudes
  e.bo = (e.bo + 1.1e-7f * na + 3e-6f * sa) * 1.001f;
}

// a lane's contribution to the change of the action from its estimates, in
// units of tau g / 2: the old terms raise it, the new ones raise (sgn_new = 1,
// the reference's rules for a swap) or lower it, and a bound that covers the
// FP32 accumulation (two ulp a term) and the sums over a warp and 16 warps
__device__ __forceinline__ void est_lane(const PairEst &q, float sgn_new, float &t, float &r) {
  t = fmaf(sgn_new, q.sn, q.so);
  const float ro = 2.4e-7f * (float)(q.ko + 1), rn = 2.4e-7f * (float)(q.kn + 1);
  const float ao = fabsf(q.so), an = fabsf(q.sn);
  r = (q.bo * (1.f + ro) + ro * ao + q.bn * (1.f + rn) + rn * an + 2e-6f * (ao + an)) * 1.00001f + 1e-30f;
}

// the Metropolis decision of a log ratio known to lie in [s - r, s + r], from
// lu = log u: 1 accept, 0 reject, -1 undecided.  The margin covers logf and
// the roundings of u, s and r (floats: 6e-8 each); lu = -inf is undecided.
__device__ __forceinline__ int decide_f(float s, float r, float lu) {
  const float mg = r * 1.00001f + 1e-5f * (1.f + fabsf(lu)) + 1e-6f * fabsf(s);
  if (s - mg > lu && lu > -3e38f) return 1;
  if (s + mg < lu) return 0;
  return -1;
}

}  // namespace pimc
