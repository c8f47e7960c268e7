// pimc_fused.cu -- the fused sweep kernels (every phase of a sweep in one
// launch; one CTA or one warp per chain), in a translation unit of their own
// so that they compile in parallel with the rest.
#include <cuda_runtime.h>

#include "pimc_sweep.cuh"

namespace pimc {

// one CTA per chain, every phase of the sweep in one launch
__global__ void __launch_bounds__(512, 1) k_sweep(SweepArgs a) { sweep_cta<SW_ALL, SWAP_LISTS>(a); }
// the same for CTAs of up to 256 threads with up to 255 registers a thread: no
// spills in the pair scans, where shared memory or the number of chains keeps
// a second CTA off the SM anyway
__global__ void __launch_bounds__(256, 1) k_sweep_wide(SweepArgs a) { sweep_cta<SW_ALL, SWAP_LISTS>(a); }
// one warp per chain, every phase
__global__ void __launch_bounds__(256, 2) k_sweep_warp(SweepArgs a) { sweep_warp<SW_ALL>(a); }

cudaError_t launch_sweep(const SweepArgs &a, int mode, int grid, int block, size_t smem,
                         cudaStream_t s) {
  if (mode == 1) k_sweep_warp<<<grid, block, smem, s>>>(a);
  else if (mode == 2) k_sweep_wide<<<grid, block, smem, s>>>(a);
  else k_sweep<<<grid, block, smem, s>>>(a);
  return cudaGetLastError();
}
cudaError_t sweep_set_smem(int mode, size_t smem) {
  if (mode == 1)
    return allow_smem((const void *)k_sweep_warp, smem);
  const cudaError_t e = allow_smem((const void *)k_sweep_wide, smem);
  if (e != cudaSuccess) return e;
  return allow_smem((const void *)k_sweep, smem);
}
cudaError_t sweep_occupancy(int mode, int block, size_t smem, int *blocks_per_sm) {
  if (mode == 1)
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_sweep_warp, block, smem);
  if (mode == 2)
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_sweep_wide, block, smem);
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_sweep, block, smem);
}
PIMC_UNIT_ACCESSORS(fused)

}  // namespace pimc
