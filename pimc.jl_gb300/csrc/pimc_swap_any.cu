// pimc_swap_any.cu -- the swap-phase kernels for any rules (physical ratio, hard
// core, contact table), in a translation unit of their own; reached through
// pimc_swap.cu's launcher.
#include <cuda_runtime.h>

#include "pimc_sweep.cuh"

namespace pimc {

// one CTA per chain
__global__ void __launch_bounds__(512, 1) k_sweep_swap(SweepArgs a) { sweep_cta<SW_SWAP>(a); }
// the register variants of pimc_swap.cu
__global__ void __launch_bounds__(64, 6) k_sweep_swap_r170(SweepArgs a) { sweep_cta<SW_SWAP>(a); }
__global__ void __launch_bounds__(64, 4) k_sweep_swap_r255(SweepArgs a) { sweep_cta<SW_SWAP>(a); }
__global__ void __launch_bounds__(256, 1) k_sweep_swap_lone(SweepArgs a) { sweep_cta<SW_SWAP>(a); }
// one warp per chain: twice the chains in flight of a two-warp CTA per chain
// at the same registers per SM
__global__ void __launch_bounds__(256, 2) k_sweep_swap_warp(SweepArgs a) { sweep_warp<SW_SWAP>(a); }

const void *swap_any_kernel(int warp, int regs) {
  if (warp) return (const void *)k_sweep_swap_warp;
  if (regs == SWAP_LONE) return (const void *)k_sweep_swap_lone;
  if (regs == 170) return (const void *)k_sweep_swap_r170;
  if (regs == 255) return (const void *)k_sweep_swap_r255;
  return (const void *)k_sweep_swap;
}

PIMC_UNIT_ACCESSORS(swap_any)

}  // namespace pimc
