// pimc_sweep.cu -- kernels of the GB300 sweep engine.
//
// One CTA (or one warp) owns one chain for the duration of a sweep, of a
// block of sweeps, or of one phase of a sweep (staging, swaps, the rest as
// three launches).  Chains that fit are staged in shared memory (x, V, the
// 16-bit position mirror and next); larger ones are updated in place in
// HBM/L2.  The same kernels serve the plain path (one launch per chain) and
// the batched path (persistent grid pulling chains from a device work queue
// in LPT order, captured in a CUDA graph).  Also here: the layout
// transposes, init_world, the estimators' launch, the adjoint, the contact
// table and the FP64 throughput probe.
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>

#include "pimc_sweep.cuh"

namespace pimc {

// the sweep's phases as separate launches (staging, swaps, the rest), each
// compiled and scheduled on its own: every chain of the batch finishes one
// phase before any starts the next, so the longest chain of each phase, not
// the longest sum over phases, sets a sweep's time
__global__ void __launch_bounds__(512, 1) k_sweep_stage(SweepArgs a) { sweep_cta<SW_STAGE>(a); }
__global__ void __launch_bounds__(512, 1) k_sweep_rest(SweepArgs a) { sweep_cta<SW_REST>(a); }

// Slots of long chains (stage_long), with cell lists of the slot's own slices: its
// windows query the slices st .. st + len - 1 and no other slot's do.  Every window
// with a pair action goes to the CTA as a team, hard cores too.  Sparse chains with a
// hard core and a pair action, staging of a sweep by the short chains' walk / by this:
// 256 particles 4.80 / 5.16 ms, 512 15.0 / 12.1 (kLongPairs), 1024 58.6 / 37.0; exact
// decisions 512 4.90 / 5.15, 1024 14.4 / 13.5 (kLongTeam); hard core alone 512 8.2 / 8.7,
// 1024 24.0 / 24.3, 2048 77.7 / 76.6 (kLongHard); kLongSlots beside its figures.
// slot_lists: whether the slot's lists are usable (built by the CTA in smem).
static __device__ __forceinline__ bool slot_lists(const CV &c, SmemCtl &sc, ChainVar *var, int st, int len,
                                                  unsigned char *smem, int budget, int *ipool) {
  const ChainDesc &d = *c.d;
  if (d.cl_nc <= 0 || d.cl_mode <= 0 || sc.v.cl_hold > 0) return false;
  if (threadIdx.x == 0) {
    sc.iflag[5] = 0;
    sc.cl.bind(d, ipool);
  }
  __syncthreads();
  cells_build<false>(c, sc.cl, (int *)smem, budget / 4, &sc.iflag[5], st, len);
  __syncthreads();
  const bool use = 2 * sc.iflag[5] >= len;
  if (!use && threadIdx.x == 0) atomicMax(&var->cl_hold, kCellHold);  // as build_lists holds them off
  __syncthreads();
  return use;
}
// the walk; returns the calling thread's attempts, accepts and beads
static __device__ __forceinline__ int3 walk_long_slot(const CV &c, unsigned long long sweep, unsigned item0, int ell,
                                                      int st, int len, unsigned char *smem, int warp_scratch_d) {
  const ChainDesc &d = *c.d;
  const int tid = threadIdx.x, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const bool team = (d.flags & PF_PAIR) && (d.flags & PF_PHYS) && nwarps > 1;
  const Team tm{warp, nwarps, 1};
  int3 t = make_int3(0, 0, 0);
  for (int n = 0; n < c.N && (team || warp == 0); ++n) {
    GenDraws dr = gen_draws(make_stream(d, sweep, PH_STAGE, item0 + n));
    const int m = min(len, 2 + (int)(dr.s.uni(DRAW_CHOICE) * (ell - 1)));
    const int r = team ? window_team<true>(c, tm, n, st, m, dr, (double *)smem, warp_scratch_d)
                       : window_warp(c, n, st, m, dr, false, (double *)smem, nullptr);
    if (tid == 0) {
      t.x += 1;
      t.y += r == RES_ACCEPT;
      if (r != RES_HARDCORE) t.z += m - 1;
    }
  }
  return t;
}

// Staging with a CTA per (chain, slot): the slots of a phase share only their
// fixed boundary slices, so they run on as many SMs as there are slots.  For
// chains whose windows depend on one another (each slot a serial walk), and
// for every chain of a launch too small to fill the GPU with whole chains.
// Items in chain order (longest first), a.stage_slots per chain, the ones past
// a chain's own slots empty.  The slots add their counts to the chain's tally;
// k_stage_close adds them to the chain's counters and adapts the window length
// (close_phase) once every slot is done -- in a launch of its own, because the
// slots' items read the length.  A chain of 1024 particles (64 slices, four
// slots) went from 57 to 7.9 ms of staging, 512 chains of 8 to 512 particles from
// 72-89 to 8.4 ms.
// k_stage_slots_long: the chains of stage_long, the other kernel's without them (in
// one kernel their lists' code cost the short chains' walks 5 to 12 %)
template <bool LONG>
__device__ __forceinline__ void stage_slots(const SweepArgs &a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SmemCtl sc;
  __shared__ double red[256];
  __shared__ unsigned bits[(kMaxParticles + 31) / 32];
  __shared__ int s_item;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int nitems = a.nchains * a.stage_slots;
  for (int iter = 0;; ++iter) {
    if (tid == 0) s_item = a.queue ? atomicAdd(a.queue, 1) : (iter == 0 ? (int)blockIdx.x : nitems);
    __syncthreads();
    const int item = s_item;
    if (item >= nitems) break;
    const int ci = item / a.stage_slots, s = item % a.stage_slots;
    const int ch = a.order ? a.order[ci] : a.chain0 + ci;
    for (int k = tid; k < (int)(sizeof(ChainDesc) / 4); k += blockDim.x)
      reinterpret_cast<unsigned *>(&sc.d)[k] = reinterpret_cast<const unsigned *>(a.desc + ch)[k];
    for (int k = tid; k < (int)(sizeof(MixDev) / 4); k += blockDim.x)
      reinterpret_cast<unsigned *>(&sc.mix)[k] = reinterpret_cast<const unsigned *>(a.mix + ch)[k];
    if (tid == 0) {
      const ChainVar &v = a.var[ch];
      sc.v.sweep = v.sweep;
      sc.v.stage_m = v.stage_m;
      sc.v.err = v.err;
      sc.v.cl_hold = v.cl_hold;
      sc.chain = ch;
    }
    __syncthreads();
    const ChainDesc &d = sc.d;
    const int N = d.N, M = d.M, ph = a.stage_phase;
    const int ell = max(2, min(sc.v.stage_m, min(M - 1, WMAX))), k = (M + ell - 1) / ell;
    const bool serial = chain_serial_local(d);
    if (s >= k || ph >= sc.mix.staging_phases || (a.stage_par == 1 && !serial) || stage_long(d, blockDim.x) != LONG ||
        sc.v.err != 0) {
      __syncthreads();
      continue;
    }
    CV c = make_cv(&sc.d, a.dpool, a.ipool, a.upool);
    const bool ok = next_is_permutation<false>(c.next, N, bits);
    int n_att = 0, n_acc = 0;
    long long n_bead = 0;
    if (!ok) {
      if (tid == 0) a.var[ch].err = DERR_STATE;
    } else {
      const unsigned long long sweep = sc.v.sweep;
      const int o = min(M - 1, (int)(make_stream(d, sweep, PH_STAGE_OFF, (unsigned)ph).uni(0) * M));
      const int budget = (int)dyn_smem_bytes();
      // one slot, or several where a restored window length makes more slots
      // than the launch counted on
      for (int sl = s; sl < k; sl += a.stage_slots) {
        const int len = sl < k - 1 ? ell : M - (k - 1) * ell, st = (o + sl * ell) % M;
        const unsigned item0 = (unsigned)(ph * (N * k) + sl * N);
        if (len < 2) continue;
        // (short of memory for its scratch, a long chain of stage_slot's is walked)
        const bool slot = stage_by_slots(d) && SlotScratch::bytes(min(ell, M - 1) + 1, nwarps) <= (size_t)budget;
        const bool listed = LONG && slot_lists(c, sc, a.var + ch, st, len, smem, budget, a.ipool);
        if (LONG && (listed || !slot)) {
          CV cw = c;
          if (listed) cw.cl = &sc.cl;
          const int3 w = walk_long_slot(cw, sweep, item0, ell, st, len, smem, a.warp_scratch_d);
          n_att += w.x;
          n_acc += w.y;
          n_bead += w.z;
          __syncthreads();
        } else if (LONG) {
          stage_slot_call(c, sweep, item0, ell, st, len, smem, red, n_att, n_acc, n_bead);
        } else if (slot) {
          stage_slot(c, sweep, item0, ell, st, len, smem, red, n_att, n_acc, n_bead);
        } else if (!serial && ell <= TWMAX) {
          for (int n = tid; n < N; n += blockDim.x) {
            GenDraws dr = gen_draws(make_stream(d, sweep, PH_STAGE, item0 + n));
            const int m = min(len, 2 + (int)(dr.s.uni(DRAW_CHOICE) * (ell - 1)));
            n_acc += window_thread(c, n, st, m, dr, false, nullptr);
            n_att += 1;
            n_bead += m - 1;
          }
        } else {
          // a warp per window (pair-free), the first warp walking the slot (hard
          // core), or the CTA as a team on each window (contact table, exact
          // decisions)
          double *wsb = (double *)smem + (size_t)warp * a.warp_scratch_d;
          const bool team = serial && !(d.flags & PF_HARD) && nwarps > 1;
          const Team tm{warp, nwarps, 1};
          for (int n = serial ? 0 : warp; n < N; n += serial ? 1 : nwarps) {
            if (serial && !team && warp > 0) break;
            GenDraws dr = gen_draws(make_stream(d, sweep, PH_STAGE, item0 + n));
            const int m = min(len, 2 + (int)(dr.s.uni(DRAW_CHOICE) * (ell - 1)));
            const int r = team ? window_team<false>(c, tm, n, st, m, dr, (double *)smem, a.warp_scratch_d)
                               : window_warp(c, n, st, m, dr, false, wsb, nullptr);
            if (lane == 0 && (!team || warp == 0)) {
              n_att += 1;
              n_acc += r == RES_ACCEPT;
              if (r != RES_HARDCORE) n_bead += m - 1;
            }
          }
          __syncthreads();
        }
      }
    }
    __syncwarp();
    n_att = __reduce_add_sync(0xffffffffu, n_att);
    n_acc = __reduce_add_sync(0xffffffffu, n_acc);
    n_bead = __reduce_add_sync(0xffffffffu, (int)n_bead);
    if (lane) n_att = 0;
    if (n_att) {
      SlotTally *t = a.tally + ch;
      atomicAdd(&t->att, (unsigned)n_att);
      atomicAdd(&t->acc, (unsigned)n_acc);
      atomicAdd(&t->beads, (unsigned long long)n_bead);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(512, 1) k_stage_slots(SweepArgs a) { stage_slots<false>(a); }
__global__ void __launch_bounds__(512, 1) k_stage_slots_long(SweepArgs a) { stage_slots<true>(a); }

// the end of the slots' staging phases: close_phase of every chain they served
__global__ void k_stage_close(SweepArgs a) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= a.nchains) return;
  const int ch = a.order ? a.order[ci] : a.chain0 + ci;
  SlotTally *t = a.tally + ch;
  if (t->att == 0u) return;
  const MixDev &mix = a.mix[ch];
  ChainVar &v = a.var[ch];
  v.att[MV_STAGE] += t->att;
  v.acc[MV_STAGE] += t->acc;
  v.bead_updates += (double)t->beads;
  v.beads_kind[MV_STAGE] += (double)t->beads;
  if (mix.adapt) {
    int m = v.stage_m;
    adapt_slices(m, (double)t->acc / (double)t->att, mix.stage_min, mix.stage_max, mix.stage_minacc,
                 mix.stage_maxacc);
    v.stage_m = m;
  }
  *t = SlotTally{};
}

cudaError_t launch_stage_slots(const SweepArgs &a, bool lng, int grid, int block, size_t smem, cudaStream_t s) {
  if (lng) k_stage_slots_long<<<grid, block, smem, s>>>(a);
  else k_stage_slots<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_stage_close(const SweepArgs &a, cudaStream_t s) {
  k_stage_close<<<(a.nchains + 127) / 128, 128, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t stage_slots_set_smem(size_t smem) {
  const cudaError_t e = allow_smem((const void *)k_stage_slots, smem);
  return e != cudaSuccess ? e : allow_smem((const void *)k_stage_slots_long, smem);
}
cudaError_t stage_slots_occupancy(bool lng, int block, size_t smem, int *blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks_per_sm, lng ? (const void *)k_stage_slots_long : (const void *)k_stage_slots, block, smem);
}
size_t slot_scratch_bytes(int ell, int nwarps) {
  return (SlotScratch::bytes(ell + 1, nwarps) + 15) & ~(size_t)15;
}

// ---------------------------------------------------------------------------
// The measurement of a sweep in launches of its own, after the sweep: items of
// meas_group slices, so that a few long chains' N^2 M / 2 pairs spread over the
// GPU (measured in the sweep's own CTA, 17 ms of a 1024-particle chain's sweep
// and 50 of a batch of 512 chains');
// the pairs in two floats where two slices fit 64 KB of shared memory.  k_measure_plan lists the items of the chains
// that measure now (their sweep counter has just advanced), the items' sums go
// to their rows, and k_measure_close adds a chain's rows in order and records.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool measures_now(const SweepArgs &a, int ch) {
  const int every = a.mix[ch].measure_every;
  const unsigned long long sw = a.var[ch].sweep;
  return every > 0 && a.var[ch].err == 0 && sw > 0 && sw % (unsigned long long)every == 0;
}
__global__ void k_measure_plan(SweepArgs a) {
  const int ci = blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= a.nchains) return;
  const int ch = a.order ? a.order[ci] : ci;
  if (!measures_now(a, ch)) return;
  const int ng = (a.desc[ch].M + a.meas_group - 1) / a.meas_group, at = atomicAdd(a.meas_cnt, ng);
  for (int g = 0; g < ng; ++g) a.meas_list[at + g] = make_int2(ch, g);
}

__global__ void __launch_bounds__(128) k_measure_slices(SweepArgs a) {
  extern __shared__ __align__(16) float4 slices[];  // two staged slices of a.meas_staged beads, or none
  __shared__ ChainDesc d;
  __shared__ double red[256];
  __shared__ unsigned long long qbuf[4 * MEAS_RING];
  __shared__ int s_it;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (!a.meas_list && !measures_now(a, a.chain0)) return;
  const int nit = a.meas_list ? a.meas_cnt[0] : (int)gridDim.x;
  for (int iter = 0;; ++iter) {
    if (tid == 0) s_it = a.meas_list ? atomicAdd(a.meas_cnt + 1, 1) : (iter ? nit : (int)blockIdx.x);
    __syncthreads();
    const int it = s_it;
    if (it >= nit) break;
    const int2 item = a.meas_list ? a.meas_list[it] : make_int2(a.chain0, it);
    for (int k = tid; k < (int)(sizeof(ChainDesc) / 4); k += blockDim.x)
      reinterpret_cast<unsigned *>(&d)[k] = reinterpret_cast<const unsigned *>(a.desc + item.x)[k];
    __syncthreads();
    const CV c = make_cv(&d, a.dpool, a.ipool, a.upool);
    const int N = c.N, j0 = item.y * a.meas_group, j1 = min(c.M, j0 + a.meas_group);
    MeasureSums m;
    m.clear();
    const bool density = c.hist != nullptr;
    const double inv_bw = density ? 1.0 / d.dens_bw : 0.0;
    measure_beads(c, j0 * N + tid, j1 * N, 128, density, inv_bw, m);
    __syncwarp();
    if ((d.flags & PF_PAIR) && !(d.flags & PF_CONTACT)) {
      if (N <= a.meas_staged) {
        for (int j = j0; j < j1; ++j) {
          const bool wrap = j == c.M - 1;
          __syncthreads();  // the last slice's pairs are done
          for (int i = tid; i < N; i += 128) {
            const int in = wrap ? c.next[i] : i, jn = wrap ? 0 : j + 1;
            slices[i] = ff_bead(c.X(0, i, j), c.Xd(1, i, j), d.len_e);
            slices[N + i] = ff_bead(c.X(0, in, jn), c.Xd(1, in, jn), d.len_e);
          }
          __syncthreads();
          measure_pairs_ff(c, j, slices, slices + N, warp, 4, reinterpret_cast<unsigned *>(qbuf + warp * MEAS_RING), m);
        }
      } else {
        measure_pairs(c, j0 * N + warp, j1 * N, 4, qbuf + warp * MEAS_RING, m);
      }
    }
    if (d.rdf_nb > 0) measure_radial(c, j0, j1, warp, 4);
    block_sum_k<5>(m.s, red);
    block_sum_k<4>(m.f, red);
    if (tid == 0) {
      double *o = a.meas_part + 9 * (size_t)(d.meas_off + item.y);
      for (int k = 0; k < 5; ++k) o[k] = m.s[k];
      for (int k = 0; k < 4; ++k) o[5 + k] = m.f[k];
    }
    __syncthreads();
  }
}

// a warp per chain
__global__ void __launch_bounds__(128) k_measure_close(SweepArgs a) {
  const int ci = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (ci >= a.nchains) return;
  const int ch = a.order ? a.order[ci] : a.chain0 + ci;
  if (!measures_now(a, ch)) return;
  const ChainDesc &d = a.desc[ch];
  const int ng = (d.M + a.meas_group - 1) / a.meas_group;
  const double *p = a.meas_part + 9 * (size_t)d.meas_off;
  double v[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int g = lane; g < ng; g += 32)
    for (int k = 0; k < 9; ++k) v[k] += p[9 * (size_t)g + k];
  for (int k = 0; k < 9; ++k) v[k] = warp_sum(v[k]);
  if (lane == 0) {
    const CV c = make_cv(&d, a.dpool, a.ipool, a.upool);
    double out[NOBS];
    measure_out(d, v, v + 5, out);
    record_measurement(d, a.var[ch], c, out, c.hist != nullptr);
  }
}

cudaError_t launch_measure_sweep(const SweepArgs &a, int ngroups, int num_sms, cudaStream_t s) {
  if (a.meas_list) {
    cudaError_t e = cudaMemsetAsync(a.meas_cnt, 0, 2 * sizeof(int), s);
    if (e != cudaSuccess) return e;
    k_measure_plan<<<(a.nchains + 127) / 128, 128, 0, s>>>(a);
    ngroups = std::min(ngroups, 5 * num_sms);
  }
  const size_t smem = 32 * (size_t)a.meas_staged;
  const cudaError_t es = allow_smem((const void *)k_measure_slices, smem);
  if (es != cudaSuccess) return es;
  k_measure_slices<<<ngroups, 128, smem, s>>>(a);
  k_measure_close<<<(a.nchains + 3) / 4, 128, 0, s>>>(a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// state maintenance: layout transposes, init_world, cached links + mirror,
// measurements
// ---------------------------------------------------------------------------
// host layout x[d][n][j] (a batch buffer at d.host_off) -> device x[j][n][d]
__global__ void k_import(const ChainDesc *desc, double *dpool, const double *src, int chain0) {
  const ChainDesc &d = desc[chain0 + blockIdx.y];
  const size_t tot = (size_t)d.dim * d.N * d.M;
  double *x = dpool + d.x_off;
  const double *s = src + d.host_off;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t row = (size_t)d.N * d.dim;
    const size_t j = e / row, r = e % row;
    const size_t n = r / d.dim, k = r % d.dim;
    x[e] = s[(k * d.N + n) * d.M + j];
  }
}

__global__ void k_export(const ChainDesc *desc, const double *dpool, double *dst, int chain0) {
  const ChainDesc &d = desc[chain0 + blockIdx.y];
  const size_t tot = (size_t)d.dim * d.N * d.M;
  const double *x = dpool + d.x_off;
  double *o = dst + d.host_off;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < tot;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t k = e / ((size_t)d.M * d.N), r = e % ((size_t)d.M * d.N);
    const size_t n = r / d.M, j = r % d.M;
    o[e] = x[(j * d.N + n) * d.dim + k];
  }
}

// The same transposes through 32 x 32 tiles of (particle, slice), over a
// flat list of every chain's tiles (tile_off[c] = first tile of chain c), so
// that both sides are read and written in whole rows: the host layout
// x[d][n][j] in runs of 32 slices, the device layout x[j][n][d] in runs of
// 32 particles.  The host-layout side may be the caller's pinned host buffer,
// which the GPU reads and writes directly over the coherent CPU-GPU link
// (Grace-Blackwell NVLink-C2C): the copy and the transpose are one pass.
// Persistent grid; each block walks tiles t = blockIdx.x, += gridDim.x.
__device__ __forceinline__ int tile_chain(const int *tile_off, int c_lo, int c_hi, int t) {
  int lo = c_lo, hi = c_hi;  // tile_off[lo] <= t < tile_off[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_off[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

// dev: a device-layout buffer of its own, chain c at host_off (per-bead forces)
// instead of the positions in the pool; tile_off null: the tiles of chain c_lo
// alone, both buffers holding nothing else.
template <bool IMPORT>
__global__ void __launch_bounds__(256) k_transpose_tiles(const ChainDesc *desc, double *dpool,
                                                          double *host, const int *tile_off,
                                                          int c_lo, int c_hi, double *dev) {
  __shared__ double tile[2][32][33];
  const int t_begin = tile_off ? tile_off[c_lo] : 0;
  const int t_end = tile_off ? tile_off[c_hi] : ((desc[c_lo].N + 31) >> 5) * ((desc[c_lo].M + 31) >> 5);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int t = t_begin + blockIdx.x; t < t_end; t += gridDim.x) {
    const int c = tile_off ? tile_chain(tile_off, c_lo, c_hi, t) : c_lo;
    const ChainDesc &d = desc[c];
    const int N = d.N, M = d.M, dim = d.dim;
    const int tj = (M + 31) >> 5, lt = tile_off ? t - tile_off[c] : t;
    const int n0 = (lt / tj) * 32, j0 = (lt % tj) * 32;
    const int nn = min(32, N - n0), nj = min(32, M - j0);
    const long long off = tile_off ? d.host_off : 0;
    double *x = dev ? dev + off : dpool + d.x_off;
    double *hx = host + off;
    if (IMPORT) {
      // host rows (k, n): 32 consecutive slices per warp-wide read
      for (int r = w; r < dim * nn; r += 8) {
        const int k = r / nn, n = r % nn;
        if (lane < nj) tile[k][n][lane] = hx[((size_t)k * N + n0 + n) * M + j0 + lane];
      }
      __syncthreads();
      // device rows j: 32 particles x dim consecutive doubles each
      const int row = nn * dim;
      for (int q = threadIdx.x; q < nj * row; q += blockDim.x) {
        const int jj = q / row, e = q % row;
        const int n = e / dim, k = e % dim;
        x[((size_t)(j0 + jj) * N + n0) * dim + e] = tile[k][n][jj];
      }
      __syncthreads();
    } else {
      const int row = nn * dim;
      for (int q = threadIdx.x; q < nj * row; q += blockDim.x) {
        const int jj = q / row, e = q % row;
        const int n = e / dim, k = e % dim;
        tile[k][n][jj] = x[((size_t)(j0 + jj) * N + n0) * dim + e];
      }
      __syncthreads();
      for (int r = w; r < dim * nn; r += 8) {
        const int k = r / nn, n = r % nn;
        if (lane < nj) hx[((size_t)k * N + n0 + n) * M + j0 + lane] = tile[k][n][lane];
      }
      __syncthreads();
    }
  }
}

// init_world (src/system.jl:36-78): uniform start, closed Levy loop through
// M rows whose first and last rows coincide, teleport
__global__ void k_init_world(const ChainDesc *desc, double *dpool, int *ipool, int chain0) {
  const ChainDesc &d = desc[chain0 + blockIdx.y];
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= d.N) return;
  CV c = make_cv(&d, dpool, ipool, nullptr);
  const int M = d.M, dim = d.dim;
  GenDraws dr = gen_draws(make_stream(d, 0, PH_INIT, (unsigned)n));
  const double L = d.L, inv2L = 1.0 / (2.0 * L);
  double st[2] = {0.0, 0.0};
  for (int k = 0; k < dim; ++k) {
    st[k] = 2.0 * L * (dr.uniform() - 0.5);
    c.X(k, n, 0) = st[k];
    c.X(k, n, M - 1) = st[k];
  }
  const int mm = M - 2;
  double p[2] = {st[0], st[1]};
  for (int j = 1; j <= mm; ++j) {
    const double al = (double)(mm + 1 - j) / (double)(mm + 2 - j);
    const double sg = sqrt(2.0 * d.lambda * al * d.tau);
    double z[2];
    for (int k = 0; k < dim; ++k) z[k] = dr.normal();
    for (int k = 0; k < dim; ++k) {
      p[k] = al * p[k] + (1.0 - al) * st[k] + z[k] * sg;
      c.X(k, n, j) = p[k];
    }
  }
  for (int k = 0; k < dim; ++k)
    for (int j = 0; j < M; ++j) c.X(k, n, j) = teleport(c.X(k, n, j), L, inv2L);
  c.next[n] = n;
}

// init_world with a hard core (src/system.jl:44-64): one warp per chain, the
// particles in order.  Lane 0 draws a particle's start and Levy loop from the
// particle's own stream in k_init_world's order (so a particle that fits at
// once gets k_init_world's path); the warp then checks every bead against the
// beads of the earlier particles at its slice (norm of the per-component
// minimum-image distances below a).  A particle that overlaps is drawn again
// from its continuing stream, at most 10000 times, after which the chain gets
// ChainVar::err = DERR_INIT and the world is not made.
__global__ void k_init_world_hard(const ChainDesc *desc, ChainVar *var, double *dpool, int *ipool,
                                  int chain0) {
  const int ch = chain0 + blockIdx.x;
  const ChainDesc &d = desc[ch];
  if (!(d.flags & PF_HARD)) return;
  const int lane = threadIdx.x & 31;
  CV c = make_cv(&d, dpool, ipool, nullptr);
  const int N = d.N, M = d.M, dim = d.dim;
  const double L = d.L, inv2L = 1.0 / (2.0 * L);
  for (int n = 0; n < N; ++n) {
    GenDraws dr = gen_draws(make_stream(d, 0, PH_INIT, (unsigned)n));
    bool placed = false;
    for (int tries = 0; tries < 10000 && !placed; ++tries) {
      if (lane == 0) {
        double st[2] = {0.0, 0.0};
        for (int k = 0; k < dim; ++k) {
          st[k] = 2.0 * L * (dr.uniform() - 0.5);
          c.X(k, n, 0) = st[k];
          c.X(k, n, M - 1) = st[k];
        }
        const int mm = M - 2;
        double pp[2] = {st[0], st[1]};
        for (int j = 1; j <= mm; ++j) {
          const double al = (double)(mm + 1 - j) / (double)(mm + 2 - j);
          const double sg = sqrt(2.0 * d.lambda * al * d.tau);
          double z[2];
          for (int k = 0; k < dim; ++k) z[k] = dr.normal();
          for (int k = 0; k < dim; ++k) {
            pp[k] = al * pp[k] + (1.0 - al) * st[k] + z[k] * sg;
            c.X(k, n, j) = pp[k];
          }
        }
        for (int k = 0; k < dim; ++k)
          for (int j = 0; j < M; ++j) c.X(k, n, j) = teleport(c.X(k, n, j), L, inv2L);
      }
      __syncwarp();
      int hit = 0;
      for (int q = lane; q < M * n && !hit; q += 32) {
        const int j = q / n, i = q % n;
        double s2 = 0.0;
        for (int k = 0; k < dim; ++k) {
          const double dd = dist1(c.X(k, i, j), c.X(k, n, j), L);
          s2 = __dadd_rn(s2, __dmul_rn(dd, dd));
        }
        if (__dsqrt_rn(s2) < d.hard_a) hit = 1;
      }
      placed = !__any_sync(0xffffffffu, hit);
    }
    if (!placed) {
      if (lane == 0) var[ch].err = DERR_INIT;
      return;
    }
    if (lane == 0) c.next[n] = n;
    __syncwarp();
  }
}

// cached link actions V[j][n] = lnV(bead, next bead) and the 16-bit mirror
__global__ void k_links(const ChainDesc *desc, double *dpool, int *ipool, int chain0) {
  const ChainDesc &d = desc[chain0 + blockIdx.y];
  CV c = make_cv(&d, dpool, ipool, nullptr);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.N * d.M; k += gridDim.x * blockDim.x) {
    const int j = k / d.N, i = k % d.N;
    const int in = j == d.M - 1 ? c.next[i] : i, jn = j + 1 == d.M ? 0 : j + 1;
    const double ax = c.X(0, i, j), ay = c.Xd(1, i, j);
    const double bx = c.X(0, in, jn), by = c.Xd(1, in, jn);
    c.Vl(i, j) = -0.5 * d.tau * (vext(d, ax, ay) + vext(d, bx, by));
    c.xq[(size_t)j * c.ldn + i] = qpos(d, ax, ay);
  }
}

// the same over the batch's 32 x 32 (particle, slice) tiles: a warp takes four
// slices of a tile, a lane a particle, and carries the potential from slice to
// slice (five evaluations for four links instead of eight).  One grid over the
// tiles: the grid of k_links, sized by the longest chain, is three quarters
// empty blocks on uneven batches (4096 chains, upload with links 7.67 -> 6.55 ms).
__global__ void __launch_bounds__(256) k_links_tiles(const ChainDesc *desc, double *dpool, int *ipool,
                                                      const int *tile_off, int c_lo, int c_hi) {
  const int t_end = tile_off[c_hi], lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int t = tile_off[c_lo] + blockIdx.x; t < t_end; t += gridDim.x) {
    const int ch = tile_chain(tile_off, c_lo, c_hi, t);
    const ChainDesc &d = desc[ch];
    const int M = d.M, tj = (M + 31) >> 5, lt = t - tile_off[ch];
    const int n = (lt / tj) * 32 + lane, j0 = (lt % tj) * 32 + 4 * w, j1 = min(M, j0 + 4);
    if (n >= d.N || j0 >= M) continue;
    const CV c = make_cv(&d, dpool, ipool, nullptr);
    const double mhtau = -0.5 * d.tau;
    double x = c.X(0, n, j0), y = c.Xd(1, n, j0), v = vext(d, x, y);
    for (int j = j0; j < j1; ++j) {
      const int in = j == M - 1 ? c.next[n] : n, jn = j + 1 == M ? 0 : j + 1;
      const double xn = c.X(0, in, jn), yn = c.Xd(1, in, jn), vn = vext(d, xn, yn);
      c.Vl(n, j) = mhtau * (v + vn);
      c.xq[(size_t)j * c.ldn + n] = qpos(d, x, y);
      x = xn;
      y = yn;
      v = vn;
    }
  }
}

// the 16-bit mirror alone (after verbatim state uploads)
__global__ void k_mirror(const ChainDesc *desc, double *dpool, int chain0) {
  const ChainDesc &d = desc[chain0 + blockIdx.y];
  CV c = make_cv(&d, dpool, nullptr, nullptr);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < d.N * d.M; k += gridDim.x * blockDim.x) {
    const int j = k / d.N, i = k % d.N;
    c.xq[(size_t)j * c.ldn + i] = qpos(d, c.X(0, i, j), c.Xd(1, i, j));
  }
}

__global__ void __launch_bounds__(256) k_measure(const ChainDesc *desc, ChainVar *var, double *dpool,
                                                 int *ipool, unsigned long long *upool, int chain0) {
  __shared__ SmemCtl sc;
  __shared__ double red[256];
  const int ch = chain0 + blockIdx.x;
  if (threadIdx.x == 0) {
    sc.d = desc[ch];
    sc.v = var[ch];
  }
  __syncthreads();
  CV c = make_cv(&sc.d, dpool, ipool, upool);
  __shared__ unsigned long long qbuf[8 * PQ_CAP];
  __shared__ unsigned bits[(kMaxParticles + 31) / 32];
  if (sc.v.err != 0 || !next_is_permutation<false>(c.next, sc.d.N, bits)) {
    if (threadIdx.x == 0) {
      if (sc.v.err == 0) sc.v.err = DERR_STATE;
      var[ch] = sc.v;
    }
    return;
  }
  measure_group(c, red, sc.e4, c.hist != nullptr, qbuf);
  if (threadIdx.x == 0) {
    record_measurement(sc.d, sc.v, c, sc.e4, c.hist != nullptr);
    var[ch] = sc.v;
  }
}

// ---------------------------------------------------------------------------
// adjoint of the potential action S_pot = -sum lnV - sum lnU: per-bead dS/dr
// and dS/d(V0, omega, g), one chain or every chain of a batch.
//
// A pair (i, b) of slice j enters two links: the one it starts (when it is
// within reach at j) and the one it ends (when its beads one slice earlier,
// along the paths, were within reach there).  Both uses carry the same
// exponential at slice j, so k_adjoint_gather evaluates it once per pair and
// slice, times the number of uses, and gathers it into the bead: no second
// pass over the links' ends and no atomics.
//
// A warp takes `ib` particles of one slice.  For each, the lanes test 32
// partners at a time on the mirror words of slices j and j-1 (integer), push
// the ones in reach at either onto a ring in shared memory, and evaluate 32
// of them at once in FP64 -- the FP64 pipe (16 cycles of an SM per warp
// instruction, whatever the active lanes) is the bound, so its instructions
// run on full warps, compares run on the bits, and the earlier slice's reach
// is settled on the mirror unless it lies within the mirror's error of the
// cut-off.  Before, one thread per bead scanned its partners (5.6 of 32 lanes
// active in the FP64 branch) and a batch's CTA per slice added forces through
// FP64 shared atomics (compare-and-swap loops).  Whole calls: one chain of N =
// 1024, M = 64 (lattice, trap, pair) 5.97 -> 0.39 ms; 60 chains of 8 to 512
// particles with every bead's force 29.4 -> 5.3 ms, of which k_adjoint_slices
// takes 4.6 (its rare parts out of line and the weight at one rounding less: 5.9
// -> 5.3).
//
// Partial sums per CTA: part[cta][9] = S_ext, dV0, domega, S_pair, dg, pair
// virial, r.g_ext, 0, r.dS/dr.
// ---------------------------------------------------------------------------
__global__ void k_adjoint_inv(AdjArgs a) {
  const int ch = a.cta_first ? (int)blockIdx.y : a.chain;
  const ChainDesc &d = a.desc[ch];
  const int *next = a.ipool + d.next_off;
  int *inv = a.inv + (a.cta_first ? a.inv_off[ch] : 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < d.N; i += gridDim.x * blockDim.x)
    inv[next[i]] = i;
}

// the sums over the warp of eight values a lane: lane l ends with the sum of
// value l & 7 (nine FP64 additions instead of forty)
__device__ __forceinline__ double warp_sum8(const double (&v)[8]) {
  const int lane = threadIdx.x & 31;
  double a[4], b[2];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const bool up = lane & 4;
    a[q] = (up ? v[q + 4] : v[q]) + __shfl_xor_sync(0xffffffffu, up ? v[q] : v[q + 4], 4);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const bool up = lane & 2;
    b[q] = (up ? a[q + 2] : a[q]) + __shfl_xor_sync(0xffffffffu, up ? a[q] : a[q + 2], 2);
  }
  const bool up = lane & 1;
  double c = (up ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, up ? b[0] : b[1], 1);
  c += __shfl_xor_sync(0xffffffffu, c, 8);
  c += __shfl_xor_sync(0xffffffffu, c, 16);
  return c;
}

constexpr int ADJ_RING = 128;  // ring entries per warp (at most 31 + 64 in use)
// whether the pair's mirror words at a slice (ci, wc) or at the one before
// (pi, wp) may lie within reach, and its ring entry: the partner, and for the
// earlier slice 0 beyond, 1 within, 2 within the mirror's error of the cut-off
__device__ __forceinline__ bool adjoint_reach(unsigned ci, unsigned pi, unsigned wc, unsigned wp,
                                              unsigned lim_lo, unsigned lim_hi, int b, unsigned &e) {
  const unsigned d2c = qdist2(ci, wc), d2p = qdist2(pi, wp);
  const unsigned st = d2p < lim_lo ? 1u : (d2p <= lim_hi ? 2u : 0u);
  e = (unsigned)b | (st << 16);
  return d2c <= lim_hi || st;
}

// The rarely taken parts of a pair, out of line: an FP64 instruction that is
// predicated off, or that the compiler evaluates ahead of a select, costs the
// pipe as much as one that runs (inline, they took 5 of a pair's 26).
static __device__ __noinline__ double adjoint_wrap(double dx, double L2) { return dx - copysign(L2, dx); }
__device__ __forceinline__ double adjoint_sep(double a, double b, double L, double L2) {  // as mi1
  const double dx = a - b;
  return abs_gt(dx, L) ? adjoint_wrap(dx, L2) : dx;
}
static __device__ __noinline__ int adjoint_near(CV c, int i, int b, int jp, const int *inv) {
  const int ip = inv ? inv[i] : i, bp = inv ? inv[b] : b;
  return mi2(*c.d, c.X(0, ip, jp), c.Xd(1, ip, jp), c.X(0, bp, jp), c.Xd(1, bp, jp)) <= c.d->rc2;
}
static __device__ __noinline__ double adjoint_weight_far(double r2, double cg, int uses) {
  return (double)uses * exp(-r2 * cg);
}
// uses exp(-cg r2) by exp_neg's table and polynomial: the product goes into both
// its roundings (to k / 64 by adding 1.5 2^46, and to the rest, then exact but
// for one rounding), the doubling into the exponent of the table's entry.  far:
// the bits of the r2 from which the library's exp takes over.
__device__ __forceinline__ double adjoint_weight(double r2, double cg, long long far, int uses) {
  if ((unsigned long long)__double_as_longlong(r2) > (unsigned long long)far) return adjoint_weight_far(r2, cg, uses);
  const double t = fma(r2, -cg, 105553116266496.0);
  const unsigned k = min((unsigned)-__double2loint(t), (unsigned)EXPTAB_N);
  const double f = fma(r2, -cg, 105553116266496.0 - t);
  double p = fma(f, 1.0 / 120.0, 1.0 / 24.0);
  p = fma(p, f, 1.0 / 6.0);
  p = fma(p, f, 0.5);
  p = fma(p, f, 1.0);
  p = fma(p, f, 1.0);
  const double e = __ldg(&g_exptab[k]);
  return __hiloint2double(__double2hiint(e) + ((uses - 1) << 20), __double2loint(e)) * p;
}
__device__ __forceinline__ long long adjoint_far(double cg) { return __double_as_longlong(39.99 / cg); }

// the uses of a pair at slice j -- the link it starts (r2 within reach) and the
// link it ends (the earlier beads' reach, settled by the entry or exactly)
__device__ __forceinline__ int adjoint_uses(const CV &c, const ChainDesc &d, unsigned e, double r2, int i, int b,
                                            int jp, const int *inv) {
  int uses = __double_as_longlong(r2) <= __double_as_longlong(d.rc2) ? 1 : 0;
  const unsigned st = e >> 16;
  if (st == 1u) {
    ++uses;
  } else if (st == 2u) {
    uses += adjoint_near(c, i, b, jp, inv);
  }
  return uses;
}

// a bead's external terms of the adjoint: its gradient, and its shares of the
// partial sums
__device__ __forceinline__ void adjoint_ext(const ChainDesc &d, double ax, double ay, double &gx, double &gy,
                                            double (&v)[8]) {
  const double tau = d.tau;
  double ge[2];
  v[0] += tau * vext_grad(d, ax, ay, ge[0], ge[1]);
  gx = ge[0] * tau;
  gy = ge[1] * tau;
  if (d.flags & PF_LATT) {
    const double sx = sinpi(ax * d.lat_k), sy = d.dim > 1 ? sinpi(ay * d.lat_k) : 0.0;
    v[1] += tau * (sx * sx + sy * sy);
  }
  if (d.flags & PF_HARM) v[2] += tau * d.omega * (ax * ax + ay * ay);
  v[6] += ax * gx + ay * gy;
}

// the block's chain and its CTA within it; every thread calls it
__device__ __forceinline__ void adjoint_cta(const AdjArgs &a, const int *first, ChainDesc *d, int *ch_, int *lb_) {
  if (threadIdx.x == 0) {
    int ch = a.chain, lb = blockIdx.x;
    if (first) {
      int lo = 0, hi = a.nchains;  // first[lo] <= blockIdx.x < first[hi]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= (int)blockIdx.x) lo = mid; else hi = mid;
      }
      ch = lo;
      lb -= first[lo];
    }
    *ch_ = ch;
    *lb_ = lb;
    *d = a.desc[ch];
  }
  __syncthreads();
}

// the CTA's row of partial sums: four warps' v[0..7] and r.dS/dr
__device__ __forceinline__ void adjoint_part(const AdjArgs &a, const double (&v)[8], double rg, double (*red)[9]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s8 = warp_sum8(v);
  rg = warp_sum(rg);
  if (lane < 8) red[warp][lane] = s8;
  if (lane == 8) red[warp][8] = rg;
  __syncthreads();
  if (threadIdx.x < 9)
    a.part[(size_t)blockIdx.x * 9 + threadIdx.x] =
        (red[0][threadIdx.x] + red[1][threadIdx.x]) + (red[2][threadIdx.x] + red[3][threadIdx.x]);
}

// the sums over the warp of two values: lanes 0-15 end with x's, 16-31 with
// y's (five FP64 additions)
__device__ __forceinline__ double warp_sum2(double x, double y) {
  const bool up = (threadIdx.x & 16) != 0;
  double f = (up ? y : x) + __shfl_xor_sync(0xffffffffu, up ? x : y, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
  return f;
}

__global__ void __launch_bounds__(128) k_adjoint_gather(AdjArgs a) {
  __shared__ ChainDesc d;
  __shared__ int s_ch, s_lb;
  __shared__ unsigned ring_s[4][ADJ_RING];
  __shared__ double red[4][9];
  adjoint_cta(a, a.cta_first, &d, &s_ch, &s_lb);
  CV c = make_cv(&d, a.dpool, a.ipool, nullptr);
  const int N = c.N, M = c.M, dim = c.dim;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nib = (N + a.ib - 1) / a.ib, unit = s_lb * 4 + warp;
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, rg = 0.0;
  if (unit < M * nib) {
    const int j = unit / nib, i0 = (unit % nib) * a.ib, ni = min(a.ib, N - i0);
    const int jp = j ? j - 1 : M - 1;
    const int *inv = j ? nullptr : a.inv + (a.cta_first ? a.inv_off[s_ch] : 0);
    const unsigned *row = c.xq + (size_t)j * c.ldn, *rowp = c.xq + (size_t)jp * c.ldn;
    const bool own = lane < ni;
    const int me = i0 + lane;
    double ax = 0.0, ay = 0.0, gx = 0.0, gy = 0.0;
    unsigned qc = 0u, qp = 0u;
    if (own) {
      ax = c.X(0, me, j);
      ay = c.Xd(1, me, j);
      qc = row[me];
      qp = rowp[inv ? inv[me] : me];
      adjoint_ext(d, ax, ay, gx, gy, v);
    }
    if ((d.flags & PF_PAIR) && N > 1) {
      const double cg = d.inv2s2, h = 0.5 * d.tau;
      const long long far = adjoint_far(cg);
      const double kf = -2.0 * cg * h * d.g;  // the force's factor
      const unsigned lim_lo = d.q_lim_lo, lim_hi = d.q_lim_hi, lt = (1u << lane) - 1u;
      unsigned *ring = ring_s[warp];
      double se = 0.0, sr = 0.0;  // sums over ordered pairs of e and r^2 e
      for (int ii = 0; ii < ni; ++ii) {
        const int i = i0 + ii;
        const double px = __shfl_sync(0xffffffffu, ax, ii), py = __shfl_sync(0xffffffffu, ay, ii);
        const unsigned ci = __shfl_sync(0xffffffffu, qc, ii), pi = __shfl_sync(0xffffffffu, qp, ii);
        double fx = 0.0, fy = 0.0;
        int head = 0, tail = 0;
        auto eval = [&](int k) {
          if (lane < k) {
            const unsigned e = ring[(head + lane) & (ADJ_RING - 1)];
            const int b = (int)(e & 0xffffu);
            const double dx = adjoint_sep(px, c.X(0, b, j), d.L, d.L2);
            const double dy = dim > 1 ? adjoint_sep(py, c.X(1, b, j), d.L, d.L2) : 0.0;
            double r2 = dx * dx;
            if (dim > 1) r2 = fma(dy, dy, r2);
            const int uses = adjoint_uses(c, d, e, r2, i, b, jp, inv);
            if (uses) {
              const double w = adjoint_weight(r2, cg, far, uses);
              se += w;
              sr = fma(r2, w, sr);
              fx = fma(w, dx, fx);
              fy = fma(w, dy, fy);
            }
          }
          head += k;
          __syncwarp();
        };
        // two blocks of 32 partners an iteration: four loads in flight; the
        // ring then holds at most 31 + 64 entries
        for (int b0 = 0; b0 < N; b0 += 64) {
          unsigned wc[2], wp[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int b = b0 + 32 * u + lane;
            wc[u] = b < N ? row[b] : 0u;
            wp[u] = b < N ? rowp[inv ? inv[b] : b] : 0u;
          }
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int b = b0 + 32 * u + lane;
            unsigned e = 0u;
            const bool p = b < N && b != i && adjoint_reach(ci, pi, wc[u], wp[u], lim_lo, lim_hi, b, e);
            const unsigned mk = __ballot_sync(0xffffffffu, p);
            if (p) ring[(tail + __popc(mk & lt)) & (ADJ_RING - 1)] = e;
            tail += __popc(mk);
          }
          __syncwarp();
          while (tail - head >= 32) eval(32);
        }
        if (tail > head) eval(tail - head);
        if (tail > 0) {
          const double f = warp_sum2(fx, fy);
          const double tx = __shfl_sync(0xffffffffu, f, 0), ty = __shfl_sync(0xffffffffu, f, 16);
          if (lane == ii) {
            gx = fma(kf, tx, gx);
            gy = fma(kf, ty, gy);
          }
        }
      }
      // ordered pairs: half of each sum
      v[4] = 0.5 * h * se;
      v[3] = d.g * v[4];
      v[5] = 0.5 * h * (-2.0 * cg) * d.g * sr;
    }
    if (own) {
      if (a.grad) {
        double *o = a.grad + (a.cta_first ? d.host_off : 0) + ((size_t)j * N + me) * dim;
        o[0] = gx;
        if (dim > 1) o[1] = gy;
      }
      rg = dim > 1 ? fma(ay, gy, ax * gx) : ax * gx;
    }
  }
  adjoint_part(a, v, rg, red);
}

// the same adjoint with every unordered pair evaluated once, for batches with
// a CTA per (chain, slice) to spare: warp w takes the particles w, w + 4, ...
// and their partners of higher index; the force goes to the particle by a
// warp sum and to the partners through the warp's own accumulators in shared
// memory (within a round of 32 the partners differ, so plain loads and stores
// do; 64 N bytes for the four warps, summed at the end).  Half of the
// gather's evaluations, at two more FP64 operations each.
__global__ void __launch_bounds__(128) k_adjoint_slices(AdjArgs a) {
  extern __shared__ __align__(16) unsigned char dsm[];
  __shared__ ChainDesc d;
  __shared__ int s_ch, s_lb;
  __shared__ unsigned ring_s[4][ADJ_RING];
  __shared__ double red[4][9];
  adjoint_cta(a, a.cta_first, &d, &s_ch, &s_lb);
  CV c = make_cv(&d, a.dpool, a.ipool, nullptr);
  const int N = c.N, M = c.M, dim = c.dim, j = s_lb, jp = j ? j - 1 : M - 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int *inv = j ? nullptr : a.inv + (a.cta_first ? a.inv_off[s_ch] : 0);
  const unsigned *row = c.xq + (size_t)j * c.ldn, *rowp = c.xq + (size_t)jp * c.ldn;
  double2 *acc = reinterpret_cast<double2 *>(dsm) + (size_t)warp * N;
  const bool pair = (d.flags & PF_PAIR) && N > 1;
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, rg = 0.0;
  const double cg = d.inv2s2, h = 0.5 * d.tau;
  const long long far = adjoint_far(cg);
  const double kf = -2.0 * cg * h * d.g;  // the force's factor
  if (pair) {
    for (int b = lane; b < N; b += 32) acc[b] = make_double2(0.0, 0.0);
    __syncwarp();
    const unsigned lim_lo = d.q_lim_lo, lim_hi = d.q_lim_hi, lt = (1u << lane) - 1u;
    unsigned *ring = ring_s[warp];
    double se = 0.0, sr = 0.0;
    for (int i = warp; i < N; i += 4) {
      const double px = c.X(0, i, j), py = c.Xd(1, i, j);
      const unsigned ci = row[i], pi = rowp[inv ? inv[i] : i];
      double fx = 0.0, fy = 0.0;
      int head = 0, tail = 0;
      auto eval = [&](int k) {
        if (lane < k) {
          const unsigned e = ring[(head + lane) & (ADJ_RING - 1)];
          const int b = (int)(e & 0xffffu);
          const double dx = adjoint_sep(px, c.X(0, b, j), d.L, d.L2);
          const double dy = dim > 1 ? adjoint_sep(py, c.X(1, b, j), d.L, d.L2) : 0.0;
          double r2 = dx * dx;
          if (dim > 1) r2 = fma(dy, dy, r2);
          const int uses = adjoint_uses(c, d, e, r2, i, b, jp, inv);
          if (uses) {
            const double w = adjoint_weight(r2, cg, far, uses);
            se += w;
            sr = fma(r2, w, sr);
            fx = fma(w, dx, fx);
            fy = fma(w, dy, fy);
            double2 t = acc[b];
            t.x = fma(-w, dx, t.x);
            t.y = fma(-w, dy, t.y);
            acc[b] = t;
          }
        }
        head += k;
        __syncwarp();
      };
      for (int b0 = (i + 1) & ~31; b0 < N; b0 += 64) {
        unsigned wc[2], wp[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int b = b0 + 32 * u + lane;
          wc[u] = b < N ? row[b] : 0u;
          wp[u] = b < N ? rowp[inv ? inv[b] : b] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int b = b0 + 32 * u + lane;
          unsigned e = 0u;
          const bool p = b < N && b > i && adjoint_reach(ci, pi, wc[u], wp[u], lim_lo, lim_hi, b, e);
          const unsigned mk = __ballot_sync(0xffffffffu, p);
          if (p) ring[(tail + __popc(mk & lt)) & (ADJ_RING - 1)] = e;
          tail += __popc(mk);
        }
        __syncwarp();
        while (tail - head >= 32) eval(32);
      }
      if (tail > head) eval(tail - head);
      if (tail > 0) {
        const double f = warp_sum2(fx, fy);
        const double ty = __shfl_sync(0xffffffffu, f, 16);
        if (lane == 0) {
          double2 t = acc[i];
          t.x += f;
          t.y += ty;
          acc[i] = t;
        }
        __syncwarp();
      }
    }
    v[4] = h * se;
    v[3] = d.g * v[4];
    v[5] = h * (-2.0 * cg) * d.g * sr;
  }
  __syncthreads();
  const double2 *all = reinterpret_cast<const double2 *>(dsm);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    const double ax = c.X(0, i, j), ay = c.Xd(1, i, j);
    double gx, gy;
    adjoint_ext(d, ax, ay, gx, gy, v);
    if (pair) {
      const double2 t0 = all[i], t1 = all[N + i], t2 = all[2 * N + i], t3 = all[3 * N + i];
      gx = fma(kf, (t0.x + t1.x) + (t2.x + t3.x), gx);
      if (dim > 1) gy = fma(kf, (t0.y + t1.y) + (t2.y + t3.y), gy);
    }
    if (a.grad) {
      double *o = a.grad + (a.cta_first ? d.host_off : 0) + ((size_t)j * N + i) * dim;
      o[0] = gx;
      if (dim > 1) o[1] = gy;
    }
    rg += dim > 1 ? fma(ay, gy, ax * gx) : ax * gx;
  }
  adjoint_part(a, v, rg, red);
}

// totals[c][9]: the partial rows of chain c's CTAs summed
__global__ void __launch_bounds__(256) k_adjoint_totals(AdjArgs a) {
  __shared__ double red[256];
  const int ch = a.cta_first ? (int)blockIdx.x : 0;
  const int b0 = a.cta_first ? a.cta_first[ch] : 0, b1 = a.cta_first ? a.cta_first[ch + 1] : a.nctas;
  double t[8] = {0, 0, 0, 0, 0, 0, 0, 0}, r[1] = {0.0};
  for (int b = b0 + threadIdx.x; b < b1; b += blockDim.x) {
    for (int q = 0; q < 8; ++q) t[q] += a.part[(size_t)b * 9 + q];
    r[0] += a.part[(size_t)b * 9 + 8];
  }
  block_sum_k<8>(t, red);
  block_sum_k<1>(r, red);
  if (threadIdx.x == 0) {
    for (int q = 0; q < 8; ++q) a.totals[(size_t)ch * 9 + q] = t[q];
    a.totals[(size_t)ch * 9 + 8] = r[0];
  }
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------

// scratch sizes of the device move routines, for the host's shared-memory plans
size_t swap_scratch_bytes(int N, int nwarps) { return SwapScratch::bytes(N, nwarps); }
size_t com_scratch_bytes(int N, int M, int nwarps) { return ComScratch::bytes(N, M, nwarps); }
int window_scratch_doubles() { return WARP_SCRATCH_D; }

// the tables of exp_neg and sincos_turn, made once for the process (the sines in
// extended precision take longer than the rest of a small handle's creation)
struct HostTables {
  double tab[TABLE_N];
  HostTables() {
    for (int k = 0; k <= EXPTAB_N; ++k) tab[k] = std::exp(-k / 64.0);
    tab[EXPTAB_N + 1] = 0.0;
    for (int k = 0; k < TURN_N; ++k) {  // a quarter turn, and exactly 0 and 1 at its ends
      const int r = k % (TURN_N / 4), q = k / (TURN_N / 4);
      const long double a = 3.14159265358979323846264338327950288L * r / (TURN_N / 2);
      const double sn = (double)sinl(a), cs = (double)cosl(a);
      tab[TURN_AT + 2 * k] = q == 0 ? sn : (q == 1 ? cs : (q == 2 ? -sn : -cs));
      tab[TURN_AT + 2 * k + 1] = q == 0 ? cs : (q == 1 ? -sn : (q == 2 ? -cs : sn));
    }
  }
};
// to the current device, in every kernel unit
cudaError_t upload_exp_table() {
  static const HostTables made;
  const double (&tab)[TABLE_N] = made.tab;
  cudaError_t e = tu_upload_exp_table(tab, sizeof(tab));
  if (e == cudaSuccess) e = swap_upload_exp_table(tab, sizeof(tab));
  if (e == cudaSuccess) e = swap_any_upload_exp_table(tab, sizeof(tab));
  if (e == cudaSuccess) e = swap_lists_upload_exp_table(tab, sizeof(tab));
  if (e == cudaSuccess) e = fused_upload_exp_table(tab, sizeof(tab));
  if (e == cudaSuccess) e = attempt_upload_exp_table(tab, sizeof(tab));
  return e;
}

// phase kernels: 0 staging, 1 swaps (pimc_swap.cu), 2 the rest; warp = 1
// (swaps only): one warp per chain; spec = 1 (swaps in CTA mode): the
// reference-rules swap kernel
static const void *phase_kernel(int phase, int warp, int spec, int regs) {
  if (phase == 1) return swap_kernel(warp, spec, regs);
  return phase == 0 ? (const void *)k_sweep_stage : (const void *)k_sweep_rest;
}
cudaError_t launch_sweep_phase(const SweepArgs &a, int phase, int warp, int spec, int regs,
                               int grid, int block, size_t smem, cudaStream_t s) {
  if (phase == 1) return launch_swap(a, warp, spec, regs, grid, block, smem, s);
  if (phase == 0) k_sweep_stage<<<grid, block, smem, s>>>(a);
  else k_sweep_rest<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t sweep_phase_set_smem(int phase, int warp, int spec, int regs, size_t smem) {
  return allow_smem(phase_kernel(phase, warp, spec, regs), smem);
}

cudaError_t sweep_phase_occupancy(int phase, int warp, int spec, int regs, int block, size_t smem,
                                  int *blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
      blocks_per_sm, phase_kernel(phase, warp, spec, regs), block, smem);
}

size_t sweep_ctl_bytes() { return (sizeof(SmemCtl) + 15) & ~(size_t)15; }
cudaError_t launch_import(const ChainDesc *desc, double *dpool, const double *src, int chain0,
                          int nchains, size_t maxn, cudaStream_t s) {
  dim3 g((unsigned)std::min<size_t>((maxn + 255) / 256, 1024), nchains);
  k_import<<<g, 256, 0, s>>>(desc, dpool, src, chain0);
  return cudaGetLastError();
}
cudaError_t launch_export(const ChainDesc *desc, const double *dpool, double *dst, int chain0,
                          int nchains, size_t maxn, cudaStream_t s) {
  dim3 g((unsigned)std::min<size_t>((maxn + 255) / 256, 1024), nchains);
  k_export<<<g, 256, 0, s>>>(desc, dpool, dst, chain0);
  return cudaGetLastError();
}
cudaError_t launch_transpose_tiles(bool import, const ChainDesc *desc, double *dpool,
                                   double *host, const int *tile_off, int c_lo, int c_hi,
                                   int ntiles, int grid, cudaStream_t s) {
  const int g = std::max(1, std::min(grid, ntiles));
  if (import) k_transpose_tiles<true><<<g, 256, 0, s>>>(desc, dpool, host, tile_off, c_lo, c_hi, nullptr);
  else k_transpose_tiles<false><<<g, 256, 0, s>>>(desc, dpool, host, tile_off, c_lo, c_hi, nullptr);
  return cudaGetLastError();
}
cudaError_t launch_init_world(const ChainDesc *desc, double *dpool, int *ipool, int chain0,
                              int nchains, int maxN, cudaStream_t s) {
  dim3 g((maxN + 127) / 128, nchains);
  k_init_world<<<g, 128, 0, s>>>(desc, dpool, ipool, chain0);
  return cudaGetLastError();
}
cudaError_t launch_init_world_hard(const ChainDesc *desc, ChainVar *var, double *dpool, int *ipool,
                                   int chain0, int nchains, cudaStream_t s) {
  k_init_world_hard<<<nchains, 32, 0, s>>>(desc, var, dpool, ipool, chain0);
  return cudaGetLastError();
}
cudaError_t launch_links(const ChainDesc *desc, double *dpool, int *ipool, int chain0, int nchains,
                         int maxNM, cudaStream_t s) {
  dim3 g((unsigned)std::min((maxNM + 255) / 256, 1024), nchains);
  k_links<<<g, 256, 0, s>>>(desc, dpool, ipool, chain0);
  return cudaGetLastError();
}
cudaError_t launch_links_tiles(const ChainDesc *desc, double *dpool, int *ipool, const int *tile_off, int c_lo,
                               int c_hi, int ntiles, int grid, cudaStream_t s) {
  k_links_tiles<<<std::max(1, std::min(grid, ntiles)), 256, 0, s>>>(desc, dpool, ipool, tile_off, c_lo, c_hi);
  return cudaGetLastError();
}
cudaError_t launch_mirror(const ChainDesc *desc, double *dpool, int chain0, int nchains, int maxNM,
                          cudaStream_t s) {
  dim3 g((unsigned)std::min((maxNM + 255) / 256, 1024), nchains);
  k_mirror<<<g, 256, 0, s>>>(desc, dpool, chain0);
  return cudaGetLastError();
}
cudaError_t launch_measure(const ChainDesc *desc, ChainVar *var, double *dpool, int *ipool,
                           unsigned long long *upool, int chain0, int nchains, cudaStream_t s) {
  k_measure<<<nchains, 256, 0, s>>>(desc, var, dpool, ipool, upool, chain0);
  return cudaGetLastError();
}
// ---------------------------------------------------------------------------
// contact-interaction propagator table (build_prop_int, src/propagator.jl:35-89):
// T(r1, r2) = -I1 - I2 + I3 on the reference's 600 x 600 grid r = 1e-20 + i h,
// with I = (1/2pi) int_0^inf k exp(-tau k^2) w(k) (Bessel products) dk
// (Gautier et al., supplementary S28), t(k) = 1/((2/pi)(gamma + log(k/2)) - 4/g0):
//   I1: w = t^2/(1+t^2), J0(k r1) J0(k r2)
//   I2: w = t/(1+t^2),   J0(k r1) Y0(k r2) + J0(k r2) Y0(k r1)
//   I3: w = t^2/(1+t^2), Y0(k r1) Y0(k r2)
// Composite 8-point Gauss-Legendre in FP64: geometric panels from 1e-10 to 0.5
// (the log behaviour at k -> 0), then uniform panels of a quarter of the
// shortest oscillation period up to K with exp(-tau K^2) = 1e-18.  CUDA's j0 /
// y0 are library calls.
//
// With t(k) = 1/s(k), s = (2/pi)(gamma + log(k/2)) - 4/g0, the weights
// t^2/(1+t^2) = wa = 1/(1+s^2) and t/(1+t^2) = wb = s/(1+s^2) stay finite where
// t has its pole, and the integrand factors over the two radii:
//   -wa J1 J2 - wb (J1 Y2 + J2 Y1) + wa Y1 Y2 = Y1 U2 + J1 V2,
//   U = wa Y - wb J, V = -(wa J + wb Y).
// So the n K distinct Bessel arguments are evaluated once (k_contact_nodes)
// and the table is the product [Y J]^T [U V] over the nodes
// (k_contact_product).  Evaluating the four functions per (entry, node)
// instead took 529 ms for n = 600, K = 4656 nodes (180300 entries, 3.4 G
// function values); the factored form has 5.6 M of them and 1.7 G FP64 FMAs,
// which the FP64 pipe (2 lanes per SM clock) bounds at 2.9 ms; the whole
// call, copy to the host included, takes 4.7 ms.
// ---------------------------------------------------------------------------
struct ContactQuad {
  double tau, g0, K, k0, du;
  int ngraded, nuniform;
};

// node q of the rule: the wave number and its weight
__device__ __forceinline__ void contact_node(const ContactQuad &c, long long q, double &k, double &w) {
  const double xs[4] = {0.18343464249564978, 0.525532409916329, 0.7966664774136267, 0.9602898564975362};
  const double ws[4] = {0.36268378337836166, 0.3137066458778869, 0.22238103445337443, 0.10122853629037706};
  const int p = (int)(q >> 3), i = (int)(q >> 1) & 3;
  double a, b;
  if (p < c.ngraded) {
    a = ldexp(1e-10, p);
    b = p + 1 == c.ngraded ? c.k0 : 2.0 * a;
  } else {
    a = c.k0 + (p - c.ngraded) * c.du;
    b = c.k0 + (p - c.ngraded + 1) * c.du;
  }
  const double mid = 0.5 * (a + b), hw = 0.5 * (b - a);
  k = (q & 1) ? mid + hw * xs[i] : mid - hw * xs[i];
  w = hw * ws[i];
}

// rows of the product for nodes [q0, q0 + kc): f[r][kc][ld], r = Y, J, U, V
__global__ void __launch_bounds__(128) k_contact_nodes(double *f, int n, int ld, long long q0, int kc, double r0,
                                                        double h, ContactQuad c) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ld) return;
  const size_t plane = (size_t)kc * ld;
  for (int q = blockIdx.y; q < kc; q += gridDim.y) {
    double k, w;
    contact_node(c, q0 + q, k, w);
    const double s = (2.0 / 3.141592653589793) * (0.5772156649015329 + log(0.5 * k)) - 4.0 / c.g0;
    const double wa = w * k * exp(-c.tau * k * k) / (1.0 + s * s) / (2.0 * 3.141592653589793), wb = s * wa;
    double J = 0.0, Y = 0.0;
    if (i < n) {
      const double x = k * (r0 + i * h);
      J = j0(x);
      Y = y0(x);
    }
    const size_t at = (size_t)q * ld + i;
    f[at] = Y;
    f[plane + at] = J;
    f[2 * plane + at] = wa * Y - wb * J;
    f[3 * plane + at] = -(wa * J + wb * Y);
  }
}

// 32 x 32 tiles of the upper triangle, 64 threads of 4 x 4 entries, blockIdx.y
// a range of the nodes; part[split][ntile][32][32].  The FP64 pipe bounds it
// (16 FMAs per 4 shared-memory loads of a thread and row), so the tiles are
// small enough that little work falls on entries below the diagonal or past
// n (7 % at n = 600), and the nodes are split to fill the SMs.
constexpr int CT_T = 32, CT_K = 16;
__global__ void __launch_bounds__(64) k_contact_product(const double *f, double *part, int ld, int kc,
                                                         int per) {
  __shared__ double sa[2][CT_K][CT_T], sb[2][CT_K][CT_T];
  int ti = 0, rest = blockIdx.x;
  const int nt = ld / CT_T;
  while (rest >= nt - ti) rest -= nt - ti++;  // row ti of tiles holds nt - ti of them
  const int tj = ti + rest;
  const int tid = threadIdx.x, ty = tid >> 3, tx = tid & 7;
  const size_t plane = (size_t)kc * ld;
  const int k_lo = blockIdx.y * per, k_hi = min(kc, k_lo + per);
  double acc[4][4] = {};
  for (int k0 = k_lo; k0 < k_hi; k0 += CT_K) {
    for (int e = tid; e < 2 * CT_K * CT_T; e += 64) {
      const int r = e / (CT_K * CT_T), kk = (e / CT_T) % CT_K, col = e % CT_T;
      const bool in = k0 + kk < k_hi;
      const size_t at = (size_t)r * plane + (size_t)(k0 + kk) * ld + col;
      sa[r][kk][col] = in ? f[at + (size_t)ti * CT_T] : 0.0;
      sb[r][kk][col] = in ? f[at + 2 * plane + (size_t)tj * CT_T] : 0.0;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < CT_K; ++kk)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        double a[4], b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u] = sa[r][kk][ty + 8 * u];
          b[u] = sb[r][kk][tx + 8 * u];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) acc[u][v] = fma(a[u], b[v], acc[u][v]);
      }
    __syncthreads();
  }
  double *o = part + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (CT_T * CT_T);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) o[(ty + 8 * u) * CT_T + tx + 8 * v] = acc[u][v];
}

// the splits' tiles summed in order into both triangles; add: onto the table
// (later ranges of nodes)
__global__ void __launch_bounds__(256) k_contact_gather(const double *part, double *tab, int n, int ld,
                                                         int ntile, int nsplit, int add) {
  const int nt = ld / CT_T;
  int ti = 0, rest = blockIdx.x;
  while (rest >= nt - ti) rest -= nt - ti++;
  const int tj = ti + rest;
  for (int e = threadIdx.x; e < CT_T * CT_T; e += blockDim.x) {
    const int i1 = ti * CT_T + e / CT_T, i2 = tj * CT_T + e % CT_T;
    if (i1 > i2 || i2 >= n) continue;
    double v = add ? tab[(size_t)i1 * n + i2] : 0.0;
    for (int s = 0; s < nsplit; ++s) v += part[((size_t)s * ntile + blockIdx.x) * (CT_T * CT_T) + e];
    tab[(size_t)i1 * n + i2] = v;
    tab[(size_t)i2 * n + i1] = v;
  }
}

// the FP32 copy of a table (scan_contact): a cell's four corners together, one
// read per term
__global__ void k_contact_cells(const double *tab, float4 *cells, int n) {
  const size_t cnt = (size_t)(n - 1) * (n - 1);
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < cnt; e += (size_t)gridDim.x * blockDim.x) {
    const size_t i = e / (n - 1), j = e % (n - 1);
    const double *t = tab + i * n + j;
    cells[e] = make_float4((float)t[0], (float)t[1], (float)t[n], (float)t[n + 1]);
  }
}
// *last: the largest index c such that an entry (c, j >= c) or (j, c) is not
// below thr in magnitude (starts at -1)
__global__ void k_contact_last(const double *tab, int n, double thr, int *last) {
  int c = -1;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * n;
       e += (size_t)gridDim.x * blockDim.x)
    if (!(fabs(tab[e]) < thr)) c = max(c, min((int)(e / n), (int)(e % n)));
  c = __reduce_max_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c >= 0) atomicMax(last, c);
}
cudaError_t launch_contact_cells(const double *tab, float4 *cells, int n, double thr, int *last, cudaStream_t s) {
  const size_t cnt = (size_t)(n - 1) * (n - 1);
  const unsigned grid = (unsigned)std::min<size_t>((cnt + 255) / 256, 1024);
  k_contact_cells<<<grid, 256, 0, s>>>(tab, cells, n);
  k_contact_last<<<grid, 256, 0, s>>>(tab, n, thr, last);
  return cudaGetLastError();
}

cudaError_t launch_contact_table(double *dtab, int n, double range, double g0, double tau,
                                 cudaStream_t s) {
  ContactQuad q;
  q.tau = tau;
  q.g0 = g0;
  q.K = sqrt(41.5 / tau);
  q.k0 = 0.5;
  q.ngraded = 33;  // 1e-10 * 2^32 > 0.5
  // the Bessel products oscillate with period >= 2 pi / (2 range): quarter
  // periods per panel
  const double period = 2.0 * 3.141592653589793 / (2.0 * range);
  const double nu = ceil((q.K - q.k0) / (0.25 * period));
  if (!(nu < 2147483600.0)) return cudaErrorInvalidValue;  // more panels than an int counts
  q.nuniform = nu < 1.0 ? 1 : (int)nu;
  q.du = (q.K - q.k0) / q.nuniform;
  const double r0 = 1e-20, h = (range - r0) / (n - 1);
  const long long nodes = 8 * ((long long)q.ngraded + q.nuniform);
  const int ld = (n + CT_T - 1) / CT_T * CT_T, nt = ld / CT_T, ntile = nt * (nt + 1) / 2;
  // about 3000 tile products in flight (ten CTAs of 64 threads per SM and a
  // second wave), never fewer than 64 nodes each
  const int nsplit = std::max(1, std::min({3000 / ntile, (int)std::min<long long>((nodes + 63) / 64, 64)}));
  const size_t npart = (size_t)nsplit * ntile * CT_T * CT_T;
  // ranges of nodes whose four rows fit a scratch of 128 MB, less when the
  // device has no such room left
  double *ws = nullptr;
  int kc = 0;
  cudaError_t e = cudaErrorMemoryAllocation;
  for (size_t room = (size_t)128 << 20; room >= ((size_t)1 << 18) && e == cudaErrorMemoryAllocation; room >>= 1) {
    kc = (int)std::min<size_t>((size_t)nodes, std::max<size_t>(CT_K, room / (32 * (size_t)ld)));
    e = cudaMalloc(&ws, 8 * (4 * (size_t)kc * ld + npart));
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  double *part = ws + 4 * (size_t)kc * ld;
  for (long long q0 = 0; q0 < nodes && e == cudaSuccess; q0 += kc) {
    const int m = (int)std::min<long long>(kc, nodes - q0);
    const int per = ((m + nsplit - 1) / nsplit + CT_K - 1) / CT_K * CT_K;
    k_contact_nodes<<<dim3((ld + 127) / 128, std::min(m, 4096)), 128, 0, s>>>(ws, n, ld, q0, m, r0, h, q);
    k_contact_product<<<dim3(ntile, nsplit), 64, 0, s>>>(ws, part, ld, m, per);
    k_contact_gather<<<ntile, 256, 0, s>>>(part, dtab, n, ld, ntile, nsplit, q0 > 0);
    e = cudaGetLastError();
  }
  const cudaError_t es = cudaStreamSynchronize(s);
  cudaFree(ws);
  return e != cudaSuccess ? e : es;
}

// ---------------------------------------------------------------------------
// FP64 pipe throughput probe: eight independent DFMA chains per thread
// ---------------------------------------------------------------------------
static __device__ double g_fp64_sink[256];

__global__ void __launch_bounds__(256) k_fp64_peak(int iters, double b, double c) {
  double a[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = 1.0 + 1e-3 * k + 1e-9 * threadIdx.x;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 8; ++k) a[k] = fma(a[k], b, c);
  }
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += a[k];
  if (s == -1.0) g_fp64_sink[threadIdx.x] = s;  // never true; keeps the chains live
}

cudaError_t fp64_peak(int num_sms, cudaStream_t st, double *tflops) {
  const int iters = 1 << 14, blocks = num_sms * 8, threads = 256;
  cudaEvent_t e0, e1;
  cudaError_t e = cudaEventCreate(&e0);
  if (e != cudaSuccess) return e;
  e = cudaEventCreate(&e1);
  if (e != cudaSuccess) {
    cudaEventDestroy(e0);
    return e;
  }
  float best = 1e30f;
  for (int rep = 0; rep < 4 && e == cudaSuccess; ++rep) {
    cudaEventRecord(e0, st);
    k_fp64_peak<<<blocks, threads, 0, st>>>(iters, 0.9999999, 1e-7);
    cudaEventRecord(e1, st);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    if (e == cudaSuccess && rep > 0 && ms < best) best = ms;  // rep 0 warms up
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e != cudaSuccess) return e;
  const double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
  *tflops = flops / (best * 1e-3) / 1e12;
  return cudaSuccess;
}

// ---------------------------------------------------------------------------
// adjoint scratch in static device memory (pimc_adjoint_noalloc): room for a
// chain of up to kNoAllocBeads beads and kNoAllocParticles particles in the
// layout of the allocating adjoint (dS/dr in both layouts, partials, totals,
// inverse permutation), 3.2 MB per device
// ---------------------------------------------------------------------------
static __device__ __align__(256) double g_adj_static[kNoAllocDoubles];

// The array's device address, per device, in an atomic slot.  Handle
// creation takes it (with the handle's device current: the set-up) and every
// later creation on that device takes it again, so the slot always holds the
// address in the device's current context: a cudaDeviceReset destroys the
// handles made before it, and the first handle made after it refreshes the
// slot before any call can use it.  Concurrent set-ups store the same value;
// readers never see a half-written entry.
namespace {
constexpr int kMaxDevices = 64;
std::atomic<double *> g_adj_addr[kMaxDevices];
}  // namespace

cudaError_t adjoint_static_setup() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  void *p = nullptr;
  e = cudaGetSymbolAddress(&p, g_adj_static);
  if (e != cudaSuccess) return e;
  g_adj_addr[dev].store(static_cast<double *>(p), std::memory_order_release);
  return cudaSuccess;
}

cudaError_t adjoint_static_scratch(double **ptr) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  double *a = g_adj_addr[dev].load(std::memory_order_acquire);
  if (!a) {
    e = adjoint_static_setup();
    if (e != cudaSuccess) return e;
    a = g_adj_addr[dev].load(std::memory_order_acquire);
  }
  *ptr = a;
  return cudaSuccess;
}

// the PIMC_PROFILE build's swap counters (g_prof of every kernel unit,
// summed): read, then cleared on request; cudaErrorNotSupported in other
// builds
cudaError_t profile_take(unsigned long long *out, bool reset, cudaStream_t s) {
#if PIMC_PROFILE
  for (int k = 0; k < 32; ++k) out[k] = 0;
  cudaError_t e = tu_profile_take(out, reset, s);
  if (e == cudaSuccess) e = swap_profile_take(out, reset, s);
  if (e == cudaSuccess) e = swap_any_profile_take(out, reset, s);
  if (e == cudaSuccess) e = swap_lists_profile_take(out, reset, s);
  if (e == cudaSuccess) e = fused_profile_take(out, reset, s);
  if (e == cudaSuccess) e = attempt_profile_take(out, reset, s);
  return e;
#else
  (void)out;
  (void)reset;
  (void)s;
  return cudaErrorNotSupported;
#endif
}

// the PIMC_CHECK build's device check word of every kernel unit (the first
// nonzero): read and cleared (0 in the default build, which has no bounds
// checks)
cudaError_t check_word_take(cudaStream_t s, unsigned long long *w) {
  cudaError_t (*const take[5])(cudaStream_t, unsigned long long *) = {
      swap_check_word_take, swap_any_check_word_take, swap_lists_check_word_take, fused_check_word_take,
      attempt_check_word_take};
  cudaError_t e = tu_check_word_take(s, w);
  for (int u = 0; u < 5 && e == cudaSuccess; ++u) {
    unsigned long long w2 = 0;
    e = take[u](s, &w2);
    if (*w == 0) *w = w2;
  }
  return e;
}

// ADJ_SLICES (a CTA per slice, every pair once) when the slices give every SM
// at least four CTAs and the accumulators of the largest chain fit the shared
// memory; else the gather, with as many particles per warp as still make
// sixteen warps per SM, from 32 down to 8, so that a small chain spreads over
// the SMs
int adjoint_ib(long long slices, long long rows32, int maxN, int num_sms, int max_dyn_smem) {
  if (slices >= 4LL * num_sms && 64LL * maxN + 8192 <= max_dyn_smem) return ADJ_SLICES;
  const long long want = 16LL * num_sms;
  return rows32 >= want ? 32 : (2 * rows32 >= want ? 16 : 8);
}

cudaError_t launch_adjoint(const AdjArgs &a, int maxN, const int *tile_off, int ntiles, double *dSdr,
                           cudaStream_t s) {
  const int nc = a.cta_first ? a.nchains : 1;
  k_adjoint_inv<<<dim3((maxN + 255) / 256, nc), 256, 0, s>>>(a);
  if (a.ib == ADJ_SLICES) {
    const size_t sm = 64 * (size_t)maxN;
    const cudaError_t e = allow_smem((const void *)k_adjoint_slices, sm);
    if (e != cudaSuccess) return e;
    k_adjoint_slices<<<a.nctas, 128, sm, s>>>(a);
  } else {
    k_adjoint_gather<<<a.nctas, 128, 0, s>>>(a);
  }
  k_adjoint_totals<<<nc, 256, 0, s>>>(a);
  if (dSdr)
    k_transpose_tiles<false><<<std::max(1, std::min(ntiles, 4096)), 256, 0, s>>>(
        a.desc, a.dpool, dSdr, tile_off, tile_off ? 0 : a.chain, tile_off ? a.nchains : a.chain + 1, a.grad);
  return cudaGetLastError();
}

}  // namespace pimc
