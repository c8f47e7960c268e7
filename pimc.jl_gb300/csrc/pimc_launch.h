// pimc_launch.h -- kernel argument blocks and host launchers of the engine.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "pimc_types.h"

namespace pimc {

// counters of a chain's slots within one sweep's staging
struct SlotTally {
  unsigned long long beads;
  unsigned att, acc;
};

struct SweepArgs {
  const ChainDesc *desc;
  ChainVar *var;
  const MixDev *mix;
  double *dpool;
  int *ipool;
  unsigned long long *upool;
  int nchains;        // chains in this launch
  int chain0;         // first chain when no queue/order is used
  const int *order;   // chain order (LPT), or null
  int *queue;         // device work-queue head, or null (one chain per CTA)
  int sweeps;         // sweeps per chain per launch
  int state_bytes;    // shared bytes reserved for staging a chain's state
  int warp_scratch_d; // doubles of scratch per warp
  int warp_bytes;     // warp-per-chain mode: scratch bytes of each warp
  int slot_bytes;     // shared bytes a CTA's slot-wise staging may use (0: none)
  int stage_par;      // k_stage_slots: 1 = only chains whose windows depend on one
                      // another (the staging kernel of whole chains has the others),
                      // 2 = every chain (lone chains, which have no such launch)
  int stage_phase;    // the staging phase that k_stage_slots runs
  int stage_slots;    // slots per chain of its queue (the longest chain's)
  struct SlotTally *tally;  // [chains] k_stage_slots' counters, zero between phases
  int measure_par;    // 1: the sweep leaves its measurement to launch_measure_sweep
  int meas_group;     // slices per item of it
  int meas_staged;    // chains of up to so many particles stage their slices
  int2 *meas_list;    // its items (chain, group), or null: chain0's groups alone
  int *meas_cnt;      // [2] items, next item
  double *meas_part;  // [items][9] partial sums (ChainDesc::meas_off)
  int teams;          // 1: staging slots walked by teams of warps (latency-bound
                      // launches whose chains all fit on the GPU at once)
};

struct AttemptArgs {
  const ChainDesc *desc;
  ChainVar *var;
  double *dpool;
  int *ipool;
  unsigned long long *upool;
  int chain, kind, n, j0, m;
  double u_pick, step;
  const double *normals;
  int n_normals;
  const double *uniforms;
  int n_uniforms;
  double *prop;
  int *out;           // result, extra, normals used, uniforms used, exhausted
  int force_warp;
};

struct EvalArgs {
  const ChainDesc *desc;
  double *dpool;
  int *ipool;
  unsigned long long *upool;
  int chain, n, j0, m;
  const double *rp;
  double *out;
};

// the adjoint of one chain (cta_first null) or of every chain of a batch: a
// warp per ib particles of a slice, four warps per CTA, chain after chain
struct AdjArgs {
  const ChainDesc *desc;
  double *dpool;
  int *ipool;
  int chain;            // the chain of a single-chain call
  int nchains;
  int ib;               // particles per warp, or ADJ_SLICES (adjoint_ib)
  int nctas;
  const int *cta_first; // [nchains + 1] first CTA of each chain, or null
  const int *inv_off;   // [nchains] offset of each chain's inverse permutation
  int *inv;             // inverse permutations
  double *part;         // [nctas][9]
  double *totals;       // [chains][9]: S_ext, dV0, domega, S_pair, dg, pair
                        // virial, r.g_ext, 0, r.dS/dr
  double *grad;         // dS/dr in the device layout [j][n][d], chains at
                        // desc.host_off (a batch) or 0, or null
};
constexpr int ADJ_SLICES = 0;  // ib: a CTA per slice instead
inline long long adjoint_ctas(int N, int M, int ib) {
  if (ib == ADJ_SLICES) return M;
  return ((long long)M * ((N + ib - 1) / ib) + 3) / 4;
}

// mode 0: one CTA per chain (k_sweep); mode 1: one warp per chain (k_sweep_warp);
// mode 2: one CTA of up to 256 threads per chain, compiled for 255 registers
cudaError_t launch_sweep(const SweepArgs &a, int mode, int grid, int block, size_t smem,
                         cudaStream_t s);
cudaError_t sweep_set_smem(int mode, size_t smem);
// the sweep as three launches per sweep (phase 0 staging, 1 swaps, 2 the
// rest), one CTA per chain, or for the swaps (warp = 1) one warp per chain;
// spec = 2 selects the swap kernels with the cell lists' bracket (swap_listed),
// spec = 1 those compiled for the reference's rules alone
// (every chain of the launch without physical rules, hard core or contact
// table); a.sweeps must be 1
// regs (swap phase in CTA mode): 0 the 128-register kernel, 170 or 255 the
// kernels compiled for CTAs of at most 64 threads with that many registers
cudaError_t launch_sweep_phase(const SweepArgs &a, int phase, int warp, int spec, int regs,
                               int grid, int block, size_t smem, cudaStream_t s);
cudaError_t sweep_phase_set_smem(int phase, int warp, int spec, int regs, size_t smem);
cudaError_t sweep_phase_occupancy(int phase, int warp, int spec, int regs, int block, size_t smem,
                                  int *blocks_per_sm);
// staging by (chain, slot) items from the work queue a.queue (a.order names
// the chains), or without one a CTA per item; lng: the chains of desc_long, else
// the others; and the end of the phases
cudaError_t launch_stage_slots(const SweepArgs &a, bool lng, int grid, int block, size_t smem, cudaStream_t s);
cudaError_t launch_stage_close(const SweepArgs &a, cudaStream_t s);
cudaError_t stage_slots_set_smem(size_t smem);
cudaError_t stage_slots_occupancy(bool lng, int block, size_t smem, int *blocks_per_sm);
// the measurement of the chains whose sweep calls for one, by (chain, slice
// group) items: of a.nchains chains in a.order, or (meas_list null) of chain
// chain0, ngroups its groups
cudaError_t launch_measure_sweep(const SweepArgs &a, int ngroups, int num_sms, cudaStream_t s);
// shared bytes of slot-wise staging for windows of at most ell slices
size_t slot_scratch_bytes(int ell, int nwarps);
size_t sweep_ctl_bytes();
cudaError_t sweep_occupancy(int mode, int block, size_t smem, int *blocks_per_sm);
cudaError_t launch_attempt(const AttemptArgs &a, size_t smem, cudaStream_t s);
cudaError_t launch_eval_action(const EvalArgs &a, cudaStream_t s);
cudaError_t launch_eval_weights(const EvalArgs &a, cudaStream_t s);
cudaError_t launch_init_world(const ChainDesc *desc, double *dpool, int *ipool, int chain0,
                              int nchains, int maxN, cudaStream_t s);
// the hard-core redraw of init_world for the chains with a hard core (one
// warp per chain; others return at once); failures set ChainVar::err
cudaError_t launch_init_world_hard(const ChainDesc *desc, ChainVar *var, double *dpool, int *ipool,
                                   int chain0, int nchains, cudaStream_t s);
cudaError_t launch_links(const ChainDesc *desc, double *dpool, int *ipool, int chain0, int nchains,
                         int maxNM, cudaStream_t s);
// the same for chains [c_lo, c_hi) over the batch's tiles (launch_transpose_tiles)
cudaError_t launch_links_tiles(const ChainDesc *desc, double *dpool, int *ipool, const int *tile_off, int c_lo,
                               int c_hi, int ntiles, int grid, cudaStream_t s);
cudaError_t launch_import(const ChainDesc *desc, double *dpool, const double *src, int chain0,
                          int nchains, size_t maxn, cudaStream_t s);
cudaError_t launch_export(const ChainDesc *desc, const double *dpool, double *dst, int chain0,
                          int nchains, size_t maxn, cudaStream_t s);
cudaError_t launch_mirror(const ChainDesc *desc, double *dpool, int chain0, int nchains, int maxNM,
                          cudaStream_t s);
// the positions of chains [c_lo, c_hi) between the host layout (at
// desc.host_off of `host`, which may be pinned host memory the GPU reaches
// directly) and the device layout, in 32 x 32 tiles; tile_off[nchains + 1]
// on the device, ntiles the range's tile count
cudaError_t launch_transpose_tiles(bool import, const ChainDesc *desc, double *dpool,
                                   double *host, const int *tile_off, int c_lo, int c_hi,
                                   int ntiles, int grid, cudaStream_t s);
cudaError_t launch_measure(const ChainDesc *desc, ChainVar *var, double *dpool, int *ipool,
                           unsigned long long *upool, int chain0, int nchains, cudaStream_t s);
int adjoint_ib(long long slices, long long rows32, int maxN, int num_sms, int max_dyn_smem);
// inverse permutations, the gather, the totals, and with dSdr (host layout,
// chains as in grad) the transpose of grad over the ntiles tiles of tile_off
// (null: one chain)
cudaError_t launch_adjoint(const AdjArgs &a, int maxN, const int *tile_off, int ntiles, double *dSdr,
                           cudaStream_t s);
cudaError_t upload_exp_table();
// PIMC_CHECK builds: the device check word (code << 32 | chain of the first
// failed bounds check, 0 if none), cleared by the read; always 0 otherwise
cudaError_t check_word_take(cudaStream_t s, unsigned long long *w);
// PIMC_PROFILE builds: the swap's section cycles [0..15] and outcome counts
// [16..31]; cudaErrorNotSupported otherwise
cudaError_t profile_take(unsigned long long *out, bool reset, cudaStream_t s);
// static adjoint scratch: kNoAllocDoubles doubles, enough for a chain of
// kNoAllocBeads beads (N*M) and kNoAllocParticles particles
constexpr int kNoAllocBeads = 65536;
constexpr int kNoAllocParticles = 8192;
constexpr size_t kNoAllocDoubles = 6 * (size_t)kNoAllocBeads +
                                   8 * (size_t)((kNoAllocBeads + 255) / 256) + 16 +
                                   (size_t)kNoAllocParticles;
// set-up: look up the array's address on the current device (every handle
// creation calls it with its device current)
cudaError_t adjoint_static_setup();
// its address on the current device, as the last set-up on it found it
cudaError_t adjoint_static_scratch(double **ptr);
// the contact-interaction propagator table T[n][n] for (range, g0, tau)
cudaError_t launch_contact_table(double *dtab, int n, double range, double g0, double tau,
                                 cudaStream_t s);
// the FP32 copy of a contact table, (n-1)^2 cells of four corners, and the last
// index whose entries reach thr (*last set to -1 before)
cudaError_t launch_contact_cells(const double *tab, float4 *cells, int n, double thr, int *last, cudaStream_t s);
// measured FP64 FMA throughput of the current device (TFLOP/s)
cudaError_t fp64_peak(int num_sms, cudaStream_t st, double *tflops);
constexpr int SWAP_LONE = 256;  // swap kernel variant for lone chains (regs)
// the swap-phase kernels' translation unit (pimc_swap.cu): its kernel for a
// launch shape and its launcher
const void *swap_kernel(int warp, int spec, int regs);
cudaError_t launch_swap(const SweepArgs &a, int warp, int spec, int regs, int grid, int block,
                        size_t smem, cudaStream_t s);
const void *swap_any_kernel(int warp, int regs);
const void *swap_lists_kernel(int regs);
// accessors of each kernel unit's device globals (swap_, swap_any_, swap_lists_, fused_, attempt_)
#define PIMC_UNIT_DECL(unit)                                                              \
  cudaError_t unit##_upload_exp_table(const double *tab, size_t bytes);                   \
  cudaError_t unit##_profile_take(unsigned long long *out, bool reset, cudaStream_t s);  \
  cudaError_t unit##_check_word_take(cudaStream_t s, unsigned long long *w);
PIMC_UNIT_DECL(swap)
PIMC_UNIT_DECL(swap_any)
PIMC_UNIT_DECL(swap_lists)
PIMC_UNIT_DECL(fused)
PIMC_UNIT_DECL(attempt)
#undef PIMC_UNIT_DECL
// shared scratch of the device move routines (bytes; doubles for a window)
size_t swap_scratch_bytes(int N, int nwarps);
size_t com_scratch_bytes(int N, int M, int nwarps);
int window_scratch_doubles();

// lets kernel f take `smem` bytes of dynamic shared memory.  The limit belongs to
// the function, not to a launch or a handle: it is only ever raised, and to all
// that the device offers, so handles on other threads never find it lowered
// between their own call and their launch.
inline cudaError_t allow_smem(const void *f, size_t smem) {
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, f);
  if (e != cudaSuccess || (size_t)fa.maxDynamicSharedSizeBytes >= smem) return e;
  int dev = 0, most = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev)) != cudaSuccess) return e;
  most -= (int)fa.sharedSizeBytes;
  if (smem > (size_t)std::max(most, 0)) return cudaErrorInvalidValue;
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

}  // namespace pimc
