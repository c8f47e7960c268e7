// pimc_swap.cu -- the swap-phase kernels of the split sweep for the reference's
// rules, and the launcher of all swap kernels; the generic ones are
// pimc_swap_any.cu's and pimc_swap_lists.cu's (translation units of their own
// compile in parallel).
#include <cuda_runtime.h>

#include "pimc_sweep.cuh"

namespace pimc {

// the swap launch for batches whose every chain follows the reference's
// rules without a hard core or a contact table (SWAP_REF), one CTA per chain
__global__ void __launch_bounds__(512, 1) k_sweep_swap_ref(SweepArgs a) {
  sweep_cta<SW_SWAP, SWAP_REF>(a);
}
// for CTAs of at most 64 threads, compiled for 6 and 4 resident CTAs per SM: up
// to 170 and 255 registers a thread instead of 128 (fewer spills, fewer chains
// in flight); and for lone chains in CTAs of up to 256 threads
__global__ void __launch_bounds__(64, 6) k_sweep_swap_ref_r170(SweepArgs a) {
  sweep_cta<SW_SWAP, SWAP_REF>(a);
}
__global__ void __launch_bounds__(64, 4) k_sweep_swap_ref_r255(SweepArgs a) {
  sweep_cta<SW_SWAP, SWAP_REF>(a);
}
__global__ void __launch_bounds__(256, 1) k_sweep_swap_ref_lone(SweepArgs a) {
  sweep_cta<SW_SWAP, SWAP_REF>(a);
}

// regs: 0 (the 128-register kernels), 170 or 255 (CTAs of 64 threads), SWAP_LONE
const void *swap_kernel(int warp, int spec, int regs) {
  if (warp || !spec) return swap_any_kernel(warp, regs);
  if (spec == 2) return swap_lists_kernel(regs);
  if (regs == SWAP_LONE) return (const void *)k_sweep_swap_ref_lone;
  if (regs == 170) return (const void *)k_sweep_swap_ref_r170;
  if (regs == 255) return (const void *)k_sweep_swap_ref_r255;
  return (const void *)k_sweep_swap_ref;
}

cudaError_t launch_swap(const SweepArgs &a, int warp, int spec, int regs, int grid, int block,
                        size_t smem, cudaStream_t s) {
  SweepArgs args = a;
  void *ptr[] = {&args};
  return cudaLaunchKernel(swap_kernel(warp, spec, regs), dim3(grid), dim3(block), ptr, smem, s);
}

PIMC_UNIT_ACCESSORS(swap)

}  // namespace pimc
