// Kernel-launch bookkeeping: every launch of this library goes through
// HB_LAUNCH so that hb_launch_count() reports how many kernels really ran.
#pragma once

#include "common.cuh"

namespace hb {
void count_launch();                 // one of this library's own kernels
void count_library_launches(int n);  // kernels launched for us by CUB

// Items (rows, ids) a warp takes per round: 32, or fewer so that a short list still fills the GPU (a
// warp moves its rows a few at a time, and 2,000 of them are 63 warps of 32).
static inline int items_per_warp(int64_t n) {
  int per = 32;
  while (per > 4 && ceil_div(n, per) < (int64_t)sm_count() * 16) per >>= 1;
  return per;
}
static inline int grid_of_warps(int64_t n, int per, int block, int blocks_per_sm) {
  int64_t blocks = ceil_div(ceil_div(n, per) * 32, block);
  const int64_t cap = (int64_t)sm_count() * blocks_per_sm;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}
}  // namespace hb

// A kernel name with template commas must be wrapped in parentheses.
#define HB_LAUNCH(kernel, grid, block, smem, stream, ...)        \
  do {                                                           \
    kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);  \
    hb::count_launch();                                          \
    HB_CUDA(cudaGetLastError());                                 \
  } while (0)
