// pimc_swap_lists.cu -- the swap-phase kernels of launches that hold long chains
// with cell lists (swap_listed), any rules: pimc_swap_any.cu's with that path, in
// a translation unit of their own.
#include <cuda_runtime.h>

#include "pimc_sweep.cuh"

namespace pimc {

__global__ void __launch_bounds__(512, 1) k_sweep_swap_lists(SweepArgs a) { sweep_cta<SW_SWAP, SWAP_LISTS>(a); }
__global__ void __launch_bounds__(64, 6) k_sweep_swap_lists_r170(SweepArgs a) { sweep_cta<SW_SWAP, SWAP_LISTS>(a); }
__global__ void __launch_bounds__(64, 4) k_sweep_swap_lists_r255(SweepArgs a) { sweep_cta<SW_SWAP, SWAP_LISTS>(a); }
__global__ void __launch_bounds__(256, 1) k_sweep_swap_lists_lone(SweepArgs a) { sweep_cta<SW_SWAP, SWAP_LISTS>(a); }

const void *swap_lists_kernel(int regs) {
  if (regs == SWAP_LONE) return (const void *)k_sweep_swap_lists_lone;
  if (regs == 170) return (const void *)k_sweep_swap_lists_r170;
  if (regs == 255) return (const void *)k_sweep_swap_lists_r255;
  return (const void *)k_sweep_swap_lists;
}

PIMC_UNIT_ACCESSORS(swap_lists)

}  // namespace pimc
