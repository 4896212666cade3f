// Kernel-launch bookkeeping: every launch of this library goes through
// HB_LAUNCH so that hb_launch_count() reports how many kernels really ran.
#pragma once

#include <utility>

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

// Entries that one cluster of CTAs sorts; more take the whole GPU (sortcore.cuh).
constexpr int64_t kSortClusterEntries = 65536;

// Captured launches do not start early: what they would give as programmatic edges of a graph was not measured.
static inline bool stream_captures(cudaStream_t st) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &c) == cudaSuccess && c != cudaStreamCaptureStatusNone;
}

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// First statement of a kernel that HB_LAUNCH_NEXT launches: everything before it in the stream is complete and seen
// from here on.  What it launches in advance is the kernel behind this one, once every block of this one has begun.
// Such a kernel lives while the one before it writes, and read-only loads are for data that nothing writes while the
// kernel lives; nor do they, or accesses through unaliased parameters, have to stay behind the wait.  So neither
// __ldg nor __restrict__ parameters in these kernels and what they call, but for load_settled.
// A kernel that runs long and leaves room on the GPU waits first and starts the next one late: blocks that wait take
// the room of kernels of other streams (three small ones beside a step of 280,000 ids, whose next launch waited
// through the sort: 98 us, now 18, as without early starts; beside an aggregation of 60,000 rows 36, now 23).
__device__ __forceinline__ void begin_after_previous() {
  wait_for_previous();
  start_next();
}

// A read-only load of what the launch before this one does not write, where that launch is always of the same call:
// it began behind all that came before it, so that nothing writes the data while this kernel lives.  (Plain loads
// are not moved up over the stores of the rows before: 100,000 inserted rows 33.9 -> 35.8 us, the expansion of 65,536
// 20.4 -> 21.1.)
template <class T>
__device__ __forceinline__ T load_settled(const T* p) { return __ldg(p); }

template <class... P, class... A>
cudaError_t launch_next(bool early, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = early && !stream_captures(st) ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // (reported here, not by the next launch of somebody else)
  return e;
}
#endif
}  // namespace hb

// A kernel name with template commas must be wrapped in parentheses.
#define HB_LAUNCH(kernel, grid, block, smem, stream, ...)        \
  do {                                                           \
    kernel<<<(grid), (block), (smem), (stream)>>>(__VA_ARGS__);  \
    hb::count_launch();                                          \
    HB_CUDA(cudaGetLastError());                                 \
  } while (0)

// A launch whose blocks may take their places while the kernel before it in the stream still runs: they wait in
// begin_after_previous.  (What the stream waits for in between, as an event of another stream, comes first as ever.)
// Steps of 2,000 to 65,536 ids are chains of five or six kernels of 3 to 35 us that had 1.7 us
// from the end of one to the start of the next (a step of 2,000 x 64 57.0 -> 49.4 us, of 65,536 x 128 130 -> 118, the
// update of 60,000 rows for Adam 87 -> 81, a round of the cold cache 171 -> 164).
#define HB_LAUNCH_NEXT_IF(early, kernel, grid, block, smem, stream, ...)                        \
  do {                                                                                          \
    HB_CUDA(hb::launch_next((early), kernel, (grid), (block), (smem), (stream), __VA_ARGS__));  \
    hb::count_launch();                                                                         \
  } while (0)
#define HB_LAUNCH_NEXT(kernel, grid, block, smem, stream, ...) \
  HB_LAUNCH_NEXT_IF(true, kernel, grid, block, smem, stream, __VA_ARGS__)
