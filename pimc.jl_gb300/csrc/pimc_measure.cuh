// pimc_measure.cuh -- the sweeps' measurements (src/measurement.jl:45-55,
// 92-122, and the radial distribution and superfluid estimators its TODOs
// name, 125-127): E_th, E_v, pair energy, pair virial, winding, area, sum r^2,
// the density and the pair-distance histogram.
//
// A link's pair within reach at its start: separations in two floats and exact
// reach, FP32 expf of both ends' squared distances (relative error about 1e-7 per
// term, far below any Monte Carlo error).  The sums of a lane's terms are exact
// to FP64 (two floats for at most 16 terms, then a double), so launch shapes
// agree to rounding.  pimc_measure keeps every term in FP64 (measure_group).
#pragma once
#include "pimc_kernels.cuh"

namespace pimc {

// a thread's sums: link, potential, virial of the external potential, pair
// energy, pair virial; winding x, y, area, sum r^2
struct MeasureSums {
  double s[5], f[4];
  __device__ void clear() {
    for (int k = 0; k < 5; ++k) s[k] = 0.0;
    for (int k = 0; k < 4; ++k) f[k] = 0.0;
  }
};

// the beads k = j N + i of k0, k0 + nt, ... below k1
__device__ __forceinline__ void measure_beads(const CV &c, int k0, int k1, int nt, bool density, double inv_bw,
                                              MeasureSums &a) {
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M, dim = c.dim;
  for (int k = k0; k < k1; k += nt) {
    const int j = k / N, i = k % N, jn = j + 1 == M ? 0 : j + 1, in = j == M - 1 ? c.next[i] : i;
    const double ax = c.X(0, i, j), ay = c.Xd(1, i, j);
    const double dx = mi1(c.X(0, in, jn), ax, d.L, d.L2);
    const double dy = dim > 1 ? mi1(c.X(1, in, jn), ay, d.L, d.L2) : 0.0;
    a.s[0] += dim > 1 ? fma(dy, dy, dx * dx) : dx * dx;
    // every bead is the start of one link and the end of another
    double gx, gy;
    a.s[1] += 2.0 * vext_grad(d, ax, ay, gx, gy);
    a.s[2] += ax * gx + (dim > 1 ? ay * gy : 0.0);
    a.f[0] += dx;
    a.f[1] += dy;
    a.f[2] += 0.5 * __dsub_rn(__dmul_rn(ax, dy), __dmul_rn(ay, dx));
    a.f[3] += __dadd_rn(__dmul_rn(ax, ax), __dmul_rn(ay, ay));
    if (density) {
      const long long ib = bin_floor(ax, d.L, d.dens_bw, inv_bw);
      bool ok = ib >= 1 && ib <= d.dens_nb;
      long long idx = ib - 1;
      if (dim > 1) {
        const long long jb = bin_floor(ay, d.L, d.dens_bw, inv_bw);
        ok = ok && jb >= 1 && jb <= d.dens_nb;
        idx += (jb - 1) * d.dens_nb;
      }
      if (ok) atomicAdd(c.hist + idx, 1ull);
    }
  }
}

// ---------------------------------------------------------------------------
// The pairs' separations in two floats (48 bits): an FP64 instruction takes one of
// the SM's four pipes for 64 cycles, the six of a pair's separations and its
// three conversions some 500 of a warp's 600 cycles; the two-float form takes
// about fifty FP32 instructions.  Its squared distance is within 2^-45, so the
// float that exp takes is the FP64 form's but for ties; a pair within 1e-6 of
// the cut-off is settled in FP64.  A measuring sweep of 4096 chains (measurement
// launches) 148 -> 51 ms.
// ---------------------------------------------------------------------------
struct FF {
  float h, l;
};
// a - b folded to the minimum image, normalised
__device__ __forceinline__ FF ff_sep(float ah, float al, float bh, float bl, float Lh, float L2h, float L2l) {
  const float s = ah - bh, z = s - ah, e = (ah - (s - z)) - (bh + z), l = e + (al - bl);
  FF r;
  r.h = s + l;
  r.l = l - (r.h - s);
  if (fabsf(r.h) >= Lh) {
    // past half the box (or within rounding of it, where the fold changes
    // nothing a pair within reach sees)
    const float f = copysignf(1.f, r.h), t = r.h - f * L2h, y = t - r.h, q = (r.h - (t - y)) + (-f * L2h - y);
    const float w = q + (r.l - f * L2l);
    r.h = t + w;
    r.l = w - (r.h - t);
  }
  return r;
}

// x 2^-len_e as two floats, the first truncated, on the integer pipe: conversions
// between the formats take the FP64 pipe's time.  Below 2^-73 of 2^len_e (which is
// no more than L, and a separation within reach is summed at L's precision) it is 0.
__device__ __forceinline__ float2 ff_bits(double x, int len_e) {
  const unsigned hi = __double2hiint(x), lo = __double2loint(x), s = hi & 0x80000000u;
  const unsigned e = (unsigned)max((int)(hi & 0x7fffffffu) - (len_e << 20), 0);
  const float h = __uint_as_float(s | __funnelshift_l(lo, e - (896u << 20), 3));
  const float u = __uint_as_float(s | (((e >> 20) - 948u) << 23));  // sign and weight of the word's last bit
  return e < (950u << 20) ? make_float2(0.f, 0.f) : make_float2(h, u * (float)(lo & 0x1fffffffu));
}

// what a chain's pairs are measured against
struct FFBox {
  float cg, Lh, L2h, L2l, r_lo, r_hi;
  int len_e;
  __device__ __forceinline__ explicit FFBox(const ChainDesc &d)
      : cg(d.inv2s2_s), Lh(d.L_s), L2h(d.L2_s), L2l(d.L2_sl), r_lo(d.rc2_s * (1.f - 1e-6f)),
        r_hi(d.rc2_s * (1.f + 1e-6f)), len_e(d.len_e) {}
  // the squared distance of beads p and r
  __device__ __forceinline__ float dist2(const float4 &p, const float4 &r) const {
    const FF dx = ff_sep(p.x, p.y, r.x, r.y, Lh, L2h, L2l), dy = ff_sep(p.z, p.w, r.z, r.w, Lh, L2h, L2l);
    const float xx = dx.h * dx.h, yy = dy.h * dy.h;
    const float ex = fmaf(dx.h, dx.h, -xx) + 2.f * dx.h * dx.l, ey = fmaf(dy.h, dy.h, -yy) + 2.f * dy.h * dy.l;
    const float s = xx + yy, z = s - xx;
    return s + (((xx - (s - z)) + (yy - z)) + (ex + ey));
  }
  // the terms of a pair within reach at r2 whose next beads are p and r: the pair
  // exponentials e = exp(x), x = -r^2/(2 s^2), and x e; the factors g tau/2 are
  // applied once at the end
  __device__ __forceinline__ void terms(float r2, const float4 &p, const float4 &r, float &e0, float &e1, float &v0,
                                        float &v1) const {
    const float nx = ff_sep(p.x, p.y, r.x, r.y, Lh, L2h, L2l).h, ny = ff_sep(p.z, p.w, r.z, r.w, Lh, L2h, L2l).h;
    const float xa = -r2 * cg, xb = -fmaf(nx, nx, ny * ny) * cg;
    const float ea = expf(xa), eb = expf(xb);
    two_sum(e0, e1, ea + eb);
    two_sum(v0, v1, fmaf(xa, ea, xb * eb));
  }
};

// a bead as two floats per coordinate
__device__ __forceinline__ float4 ff_bead(double x, double y, int len_e) {
  const float2 a = ff_bits(x, len_e), b = ff_bits(y, len_e);
  return make_float4(a.x, a.y, b.x, b.y);
}

// a pair next to the cut-off, in FP64 (out of line: a predicated FP64 instruction
// costs the pipe as much as one that runs)
static __device__ __noinline__ bool measure_near(CV c, int i, int b, int j) {
  return mi2(*c.d, c.X(0, i, j), c.Xd(1, i, j), c.X(0, b, j), c.Xd(1, b, j)) <= c.d->rc2;
}

// the pairs of a warp: rows (j, i) k = j N + i of k0, k0 + dk, ... below k1 (rows
// shorten with i: dealt to the warps in turn), the links of particles i < b that
// start at slice j.  Lanes test 32 partners on the mirror; survivors go onto a
// ring and are evaluated 32 at a time.  768 replicas of 8 to 48
// particles measured in every sweep: 3.92 -> 3.81 ms (four sweeps) by the
// separations in two floats.
constexpr int MEAS_RING = 64;  // at most 31 + 32 in use
__device__ __forceinline__ void measure_pairs(const CV &c, int k0, int k1, int dk, unsigned long long *ring,
                                              MeasureSums &a) {
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u, lim = d.q_lim_hi;
  const FFBox box(d);
  int head = 0, tail = 0, nf = 0;
  float e0 = 0.f, e1 = 0.f, v0 = 0.f, v1 = 0.f;  // running sums, high and low parts
  auto spill = [&]() {
    a.s[3] += (double)e0 + (double)e1;
    a.s[4] += (double)v0 + (double)v1;
    e0 = e1 = v0 = v1 = 0.f;
    nf = 0;
  };
  auto flush = [&](int cnt) {
    if (lane < cnt) {
      const unsigned long long w = ring[(head + lane) & (MEAS_RING - 1)];  // i | b << 13 | j << 26
      const int i = (int)(w & 0x1fffu), b = (int)((w >> 13) & 0x1fffu), j = (int)(w >> 26);
      auto bead = [&](int n, int t) { return ff_bead(c.X(0, n, t), c.Xd(1, n, t), box.len_e); };
      const float r2 = box.dist2(bead(i, j), bead(b, j));
      bool in = r2 < box.r_lo;
      if (!in && r2 <= box.r_hi) in = measure_near(c, i, b, j);
      if (in) {
        const int jn = j + 1 == M ? 0 : j + 1, in = j == M - 1 ? c.next[i] : i, bn = j == M - 1 ? c.next[b] : b;
        box.terms(r2, bead(in, jn), bead(bn, jn), e0, e1, v0, v1);
      }
    }
    head += cnt;
    __syncwarp();
    if (++nf == 16) spill();
  };
  for (int k = k0; k < k1; k += dk) {
    const int j = k / N, i = k % N;
    const unsigned *row = c.xq + (size_t)j * c.ldn;
    const unsigned ci = row[i];
    for (int b0 = i + 1; b0 < N; b0 += 32) {
      const int b = b0 + lane;
      const bool in = b < N && qdist2(ci, row[b]) <= lim;
      const unsigned mk = __ballot_sync(0xffffffffu, in);
      if (in)
        ring[(tail + __popc(mk & lt)) & (MEAS_RING - 1)] =
            (unsigned long long)((unsigned)i | ((unsigned)b << 13)) | ((unsigned long long)j << 26);
      tail += __popc(mk);
      __syncwarp();
      if (tail - head >= 32) flush(32);
    }
  }
  if (tail > head) flush(tail - head);
  spill();
}


// the pairs of slice j by a CTA of `nw` warps: cur and nxt the staged slice and
// the next along the paths; this warp takes rows w, w + nw, ...
__device__ __forceinline__ void measure_pairs_ff(const CV &c, int j, const float4 *cur, const float4 *nxt, int w,
                                                 int nw, unsigned *ring, MeasureSums &a) {
  const ChainDesc &d = *c.d;
  const int N = c.N, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u, lim = d.q_lim_hi;
  const FFBox box(d);
  int head = 0, tail = 0, nf = 0;
  float e0 = 0.f, e1 = 0.f, v0 = 0.f, v1 = 0.f;  // running sums, high and low parts
  auto spill = [&]() {
    a.s[3] += (double)e0 + (double)e1;
    a.s[4] += (double)v0 + (double)v1;
    e0 = e1 = v0 = v1 = 0.f;
    nf = 0;
  };
  auto flush = [&](int cnt) {
    if (lane < cnt) {
      const unsigned q = ring[(head + lane) & (MEAS_RING - 1)];  // i | b << 13
      const int i = (int)(q & 0x1fffu), b = (int)(q >> 13);
      const float4 p = cur[i], r = cur[b];
      const float r2 = box.dist2(p, r);
      bool in = r2 < box.r_lo;
      if (!in && r2 <= box.r_hi) in = measure_near(c, i, b, j);
      if (in) box.terms(r2, nxt[i], nxt[b], e0, e1, v0, v1);
    }
    head += cnt;
    __syncwarp();
    if (++nf == 16) spill();
  };
  const unsigned *row = c.xq + (size_t)j * c.ldn;
  for (int i = w; i < N; i += nw) {
    const unsigned ci = row[i];
    for (int b0 = i + 1; b0 < N; b0 += 32) {
      const int b = b0 + lane;
      const bool in = b < N && qdist2(ci, row[b]) <= lim;
      const unsigned mk = __ballot_sync(0xffffffffu, in);
      if (in) ring[(tail + __popc(mk & lt)) & (MEAS_RING - 1)] = (unsigned)i | ((unsigned)b << 13);
      tail += __popc(mk);
      __syncwarp();
      if (tail - head >= 32) flush(32);
    }
  }
  if (tail > head) flush(tail - head);
  spill();
}

// the pair-distance histogram of slices [j0, j1): warps gw, gw + ngw, ... over
// the beads, lanes the partners of higher index; lanes with the same bin add
// once (match_any)
__device__ __forceinline__ void measure_radial(const CV &c, int j0, int j1, int gw, int ngw) {
  const ChainDesc &d = *c.d;
  const int N = c.N, dim = c.dim, lane = threadIdx.x & 31;
  for (int kk = j0 * N + gw; kk < j1 * N; kk += ngw) {
    const int j = kk / N, i = kk % N;
    const double ax = c.X(0, i, j), ay = c.Xd(1, i, j);
    for (int b0 = i + 1; b0 < N; b0 += 32) {
      const int b = b0 + lane;
      int bin = -1;
      if (b < N) {
        const double dx = fabs(mi1(ax, c.X(0, b, j), d.L, d.L2));
        const double dy = dim > 1 ? fabs(mi1(ay, c.Xd(1, b, j), d.L, d.L2)) : 0.0;
        const double r = __dsqrt_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
        const double f = floor(r / d.rdf_dr);
        if (f < (double)d.rdf_nb) bin = (int)f;
      }
      const unsigned act = __ballot_sync(0xffffffffu, bin >= 0);
      if (bin >= 0) {
        const unsigned peers = __match_any_sync(act, bin);
        if (lane == __ffs(peers) - 1) atomicAdd(d.rdf + bin, (unsigned long long)__popc(peers));
      }
    }
  }
}

// the observables of one measurement from the chain's summed s and f
__device__ __forceinline__ void measure_out(const ChainDesc &d, const double *s, const double *f, double *out) {
  const double tau = d.tau;
  const int M = d.M;
  const bool pair = (d.flags & PF_PAIR) != 0 && !(d.flags & PF_CONTACT);
  out[4] = f[0] * f[0] + f[1] * f[1];
  out[5] = f[2];
  out[6] = f[3] / M;
  out[7] = 0.0;
  out[0] = (double)(d.dim * d.N) / (2.0 * tau) - 1.0 / (4.0 * d.lambda * (tau * tau) * M) * s[0] +
           1.0 / (2.0 * M) * s[1];
  out[1] = 1.0 / (2.0 * M) * s[2] + 1.0 / (2.0 * M) * s[1];
  // pair energy sum (tau/2) g (e_a + e_b) / (M tau) and its virial part
  // sum (tau/2) g (-2 r^2/(2 s^2)) (e_a, e_b) / (2 M tau)
  out[2] = pair ? d.g * s[3] / (2.0 * M) : 0.0;
  out[3] = pair ? out[2] + d.g * s[4] / (2.0 * M) : 0.0;
}

// a sweep's measurement by the group that sweeps the chain; qbuf: one
// PQ_CAP-entry queue per warp
template <bool WARP>
__device__ void measure_sweep(const CV &c, double *red, double *out, bool density, unsigned long long *qbuf) {
  using G = Group<WARP>;
  const ChainDesc &d = *c.d;
  const int N = c.N, M = c.M, tid = G::rank(), nt = G::size();
  const int warp = WARP ? 0 : (int)(threadIdx.x >> 5), nwarps = WARP ? 1 : (int)(blockDim.x >> 5);
  MeasureSums a;
  a.clear();
  const double inv_bw = density ? 1.0 / d.dens_bw : 0.0;
  measure_beads(c, tid, N * M, nt, density, inv_bw, a);
  __syncwarp();
  if ((d.flags & PF_PAIR) && !(d.flags & PF_CONTACT)) {
    measure_pairs(c, warp, N * M, nwarps, qbuf + (size_t)warp * PQ_CAP, a);
  }
  if (d.rdf_nb > 0) measure_radial(c, 0, M, warp, nwarps);
  G::template sum<5>(a.s, red);
  G::template sum<4>(a.f, red);
  if (tid == 0) measure_out(d, a.s, a.f, out);
}

}  // namespace pimc
