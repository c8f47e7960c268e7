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

// a lane's sums over one particle, from the mirror: e.so / e.sn old and new
// sums of exp(-r_a^2/2s^2) + exp(-r_b^2/2s^2) over the links whose start has
// the particle within reach, e.bo / e.bn bounds on their distance from the
// exact sums (a mirror distance is within kQErr units of the exact one;
// ChainDesc::est_a, est_b).  cq[t * NC + k]: mirror word of centre k at bead t,
// t = 0 .. m; word(t): the particle's; on(k): whether centre k counts it.
template <int NC, class Word, class On>
__device__ __forceinline__ void scan_block(const ChainDesc &d, int m, const unsigned *cq, const Word &word,
                                           const On &on, PairEst &e) {
  const float ca = d.est_a, cb = d.est_b, cx = d.est_x;
  unsigned lo[NC], hi[NC];
  float ep[NC], rp[NC], wp[NC], gp[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) {
    lo[k] = on(k) ? d.q_lim_lo : 0u;
    hi[k] = on(k) ? d.q_lim_hi + 1u : 0u;
    ep[k] = rp[k] = wp[k] = gp[k] = 0.f;
  }
  // the slices' words four beads ahead: a step takes a few hundred cycles, a
  // word from L2 up to a thousand
  unsigned q0 = word(0), q1 = word(min(1, m)), q2 = word(min(2, m)), q3 = word(min(3, m));
  for (int t = 0; t <= m; ++t) {
    const unsigned q = q0;
    q0 = q1;
    q1 = q2;
    q2 = q3;
    if (t + 4 <= m) q3 = word(t + 4);
#pragma unroll
    for (int k = 0; k < NC; ++k) {
      const unsigned d2 = qdist2(cq[t * NC + k], q);
      const float f = (float)d2, x = ex2_approx(f * cx);
      const float r = fmaf(x, fmaf(ca, f, cb), 1e-30f);
      const float v = ep[k] + x, ve = rp[k] + r;
      float &s = (k & 1) ? e.sn : e.so, &bd = (k & 1) ? e.bn : e.bo;
      s = fmaf(wp[k], v, s);
      bd = fmaf(wp[k], ve, bd);
      bd = fmaf(gp[k], v + ve, bd);
      ep[k] = x;
      rp[k] = r;
      // surely within reach: weight 1; unsettled: half the link, within half
      const bool in = d2 < lo[k], may = d2 < hi[k];
      gp[k] = may && !in ? 0.5f : 0.f;
      wp[k] = in ? 1.f : gp[k];
    }
  }
  e.ko += m * (NC / 2) * 3;
  e.kn += m * (NC / 2) * 3;
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
  const float u = d.f_unit, rc2 = (float)d.rc2;
  const float r_lo = rc2 * (1.f - 2e-6f) - 8.f * u * (float)d.rc, r_hi = rc2 * (1.f + 2e-6f) + 8.f * u * (float)d.rc;
  const float cy = (float)d.inv2s2;
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

// a lane's contribution to the change of the action from its estimates, in
// units of tau g / 2: the old terms raise it, the new ones raise (sgn_new = 1,
// the reference's rules for a swap) or lower it, and a bound that covers the
// FP32 accumulation (two ulp a term) and the sums over a warp and 16 warps
__device__ __forceinline__ void est_lane(const PairEst &q, float sgn_new, float &t, float &r) {
  t = fmaf(sgn_new, q.sn, q.so);
  const float ro = 2.4e-7f * (float)(q.ko + 1), rn = 2.4e-7f * (float)(q.kn + 1);
  r = (q.bo * (1.f + ro) + ro * q.so + q.bn * (1.f + rn) + rn * q.sn + 2e-6f * (q.so + q.sn)) * 1.00001f + 1e-30f;
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
