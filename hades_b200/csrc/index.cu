// Cache index in HBM: create/destroy, add, lookup, LRU touch, reset, getall,
// sorted-view build, raw export/import.  Semantics follow the reference's
// SACacheIndex (src/cache/cache.h) and cache_line (src/cache/cache_line.h);
// the data structures and kernels are new.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <cub/iterator/counting_input_iterator.cuh>

#include <chrono>
#include <thread>

#include "index.cuh"
#include "launch.cuh"
#include "maintain.cuh"
#include "sortcore.cuh"

namespace hb {
namespace {

constexpr int kBlock = 256;

__global__ void fill_i64_kernel(int64_t* p, int64_t n, int64_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void fill_i32_kernel(int32_t* p, int64_t n, int32_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

// ---- add ---------------------------------------------------------------------
// Two ways to the ids of a set in input order.
//
// (1) Sorted by set (sortcore.cuh), input order kept inside a set; one thread per set walks them.  For
//     small batches (one launch), for batches of many ids per set, and (LONG_LISTS) for the sets that
//     (2) leaves behind, usually none.
template <bool LONG_LISTS>
struct SetSource {
  static constexpr bool kSkips = LONG_LISTS;
  const int64_t* ids;
  int64_t n;
  int64_t lines;
  const unsigned long long* heads;
  const int32_t* batch;
  __host__ __device__ int known_bits() const { return 0; }
  __device__ __forceinline__ int64_t count() const { return !LONG_LISTS || batch[2] == batch[0] ? n : 0; }
  __device__ __forceinline__ bool fetch(int64_t i, int64_t& id) const {
    id = ids[i];
    return true;
  }
  __device__ __forceinline__ bool accept(int64_t id, unsigned long long& key) const {
    if (id < 0) return false;  // unusable (padding)
    key = (unsigned long long)mod_nonneg(id, lines);
    return !LONG_LISTS || heads[key] == (((unsigned long long)(uint32_t)batch[0] << 32) | kLongList);
  }
};

template <bool LONG_LISTS>
__device__ __forceinline__ void add_sorted_set(int j, int n, const uint2* kv, const int64_t* ids, int64_t* line_ids,
                                               int32_t* lru, int64_t* locs, uint8_t* last_writer) {
  const uint2 e = __ldcg(kv + j);
  if (e.x == kSortNone) {  // every thread answers for its own entry
    if (LONG_LISTS) return;
    locs[e.y] = -1;
    if (last_writer) last_writer[e.y] = 0;
    return;
  }
  if (j > 0 && __ldcg(&kv[j - 1].x) == e.x) return;  // not the head of its segment
  const int64_t line = e.x;
  LineState st;
  st.load(line_ids, lru, line);
  int k = j;
  uint2 x = e;
  while (true) {
    const int way = st.place(ids[x.y], k);
    locs[x.y] = way >= 0 ? line * kWays + way : -1;
    ++k;
    if (k >= n) break;
    x = __ldcg(kv + k);
    if (x.x != e.x) break;
  }
  st.store(line_ids, lru, line);
  if (last_writer)
    for (int m = j; m < k; ++m) {
      const uint32_t pos = __ldcg(&kv[m].y);
      last_writer[pos] = st.is_last(locs[pos], m);
    }
}

struct AddFinish {
  static constexpr bool kOneEach = false;
  int64_t* line_ids;
  int32_t* lru;
  int64_t* locs;           // [n]
  uint8_t* last_writer;    // nullable [n]: of several ids that received one slot, the last
  uint2* sorted;           // [n] scratch
  bool walk_later;         // by a launch of its own
  // nothing was placed: no slots (of the sets that the lists left behind, where only those are sorted)
  template <class Ctx, class Src>
  __device__ __forceinline__ void give_up(Ctx& ctx, const Src& src) const {
    for (uint32_t j = ctx.chunk_begin() + threadIdx.x; j < ctx.chunk_end(); j += Ctx::kThreads) {
      unsigned long long key;
      if (Src::kSkips && !sort_load(src, j, key)) continue;
      locs[j] = -1;
      if (last_writer) last_writer[j] = 0;
    }
  }
  template <class Ctx, class Src>
  __device__ __forceinline__ void run(Ctx& ctx, const Src& src) const {
    const uint2* kv = ctx.publish(sorted);
    if (walk_later) return;
    for (uint32_t j = ctx.chunk_begin() + threadIdx.x; j < ctx.chunk_end(); j += Ctx::kThreads)
      add_sorted_set<Src::kSkips>((int)j, ctx.count, kv, src.ids, line_ids, lru, locs, last_writer);
  }
};

__global__ void __launch_bounds__(kBlock) add_sorted_walk_kernel(const int64_t* ids, int n, AddFinish f) {
  const int j = blockIdx.x * kBlock + threadIdx.x;
  if (j < n) add_sorted_set<false>(j, n, f.sorted, ids, f.line_ids, f.lru, f.locs, f.last_writer);
}

// (2) Every id puts itself on the list of its set (one atomic exchange); the thread whose id ended up
//     in front owns the set, brings the list into input order and walks it.  No sort.  Lists of more
//     than 32 ids (copies of one id, ids in strides of the number of sets) go to (1).
__global__ void __launch_bounds__(kBlock) add_push_kernel(const int64_t* ids, int64_t n, AddLists lists, int64_t* locs,
                                                          uint8_t* last_writer) {
  begin_after_previous();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t id = ids[i];
  if (id >= 0) {
    lists.push(id, i);
  } else {
    locs[i] = -1;
    if (last_writer) last_writer[i] = 0;
  }
}

// the runs of a batch that are on lists, sorted by set instead (many ids per set)
struct ListedSource {
  static constexpr bool kSkips = false;
  const int64_t* ids;
  int64_t n;
  const int64_t* n_dev;
  const uint8_t* listed;
  const int64_t* cut;
  int64_t lines;
  __host__ __device__ int known_bits() const { return 0; }
  __device__ __forceinline__ int64_t count() const { return *n_dev < n ? *n_dev : n; }
  __device__ __forceinline__ bool fetch(int64_t i, int64_t& id) const {
    id = ids[i];
    return listed[i] && i < *cut;
  }
  __device__ __forceinline__ bool accept(int64_t id, unsigned long long& key) const {
    key = (unsigned long long)mod_nonneg(id, lines);
    return true;
  }
};

__global__ void __launch_bounds__(kBlock) add_cut_kernel(AddEntries e, int64_t* cut) {
  const int64_t c = add_cut<kBlock>(e, *e.n_dev < e.n ? *e.n_dev : e.n);
  if (threadIdx.x == 0) *cut = c;
}

__global__ void __launch_bounds__(kBlock) add_walk_kernel(AddEntries e, AddState a) {
  begin_after_previous();
  const uint32_t number = batch_number(a.batch);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < e.n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t id = e.ids[i];
    if (id < 0) continue;
    const int64_t line = mod_nonneg(id, a.lines);
    if (a.heads[line] != (((unsigned long long)number << 32) | (unsigned long long)(i + 1))) continue;
    LineState st;
    st.load(a.line_ids, a.lru, line);
    walk_list<false>(e, a, i, e.n, number, line, id, st);
  }
  batch_done(a.batch, number, gridDim.x);
}

// ---- lookup ------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kBlock) lookup_kernel(IndexView v, const int64_t* __restrict__ ids,
                                                         int64_t n, int64_t* __restrict__ locs,
                                                         uint8_t* __restrict__ found) {
  __shared__ int64_t s_top[MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = warp * 32; base < n; base += nwarps * 32) {
    const int64_t i = base + lane_id();
    const int64_t id = i < n ? __ldg(ids + i) : -1;
    const int64_t slot = warp_lookup<MODE>(v, s_top, id);
    if (i < n) {
      if (locs) locs[i] = slot;
      if (found) found[i] = slot >= 0;
    }
  }
}

// ---- LRU touch ---------------------------------------------------------------
// The sequential rule "all counters of the line += 1, hit way = 0" (cache_line.h:80-86) leaves after a
// whole batch
//   way hit in the batch   -> number of hits on the line after its last hit
//   way not hit            -> old counter + hits on the line
// Three passes over the batch positions, no sort: the last hit of every slot and the hits of every
// line; the hits after each slot's last; the counters.  (65,536 positions: sorted 40 us, this 9.)  Lanes
// with the same slot speak as one, so that the copies of a popular id do not queue at one address.
// A caller that works on ids in host memory has them and wants the slots in pinned buffers, a part of the
// batch at a time: positions first .. first + n of it, slots to host_locs too, and then a word that says
// that they have arrived.  Ids (as WORD, signed) and slots cross PCIe in half the bytes where the ids fit 32 bits: a
// part of 32,768 is bound by that.
template <typename WORD>
struct HostPart {
  int64_t first;
  WORD* locs;       // nullable
  int64_t* arrived; // nullable
};

template <int MODE, bool LOOKUP, typename WORD>
__global__ void __launch_bounds__(kBlock) touch_mark_kernel(IndexView v, const WORD* __restrict__ ids,
                                                            int64_t* __restrict__ locs, int64_t n, TouchMarks t,
                                                            int32_t* __restrict__ line_hits, HostPart<WORD> part) {
  __shared__ int64_t s_top[LOOKUP && MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (LOOKUP && MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  const unsigned long long number = (unsigned long long)batch_number(t.batch) << 32;
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = warp * 32; base < n; base += nwarps * 32) {
    const int64_t i = base + lane;
    int64_t slot = -1;
    if (LOOKUP) {
      slot = warp_lookup<MODE>(v, s_top, i < n ? (int64_t)__ldg(ids + i) : -1);
      if (i < n) {
        locs[i] = slot;
        if (part.locs) part.locs[i] = (WORD)slot;
      }
    } else if (i < n) {
      slot = locs[i];
      if (slot >= t.capacity) slot = -1;
    }
    const unsigned same = __match_any_sync(0xffffffffu, slot);
    if (slot >= 0 && (same >> lane) == 1u) {  // the last of them
      atomicMax(t.marks + slot, number | (unsigned long long)(part.first + i + 1));
      atomicAdd(line_hits + (slot >> 3), __popc(same));
    }
  }
  if (part.arrived) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence_system();  // after the barrier: for the stores of the whole block
      unsigned* done = reinterpret_cast<unsigned*>(t.batch + 6);
      if (atomicAdd(done, 1u) == gridDim.x - 1u) {
        *done = 0u;
        __threadfence_system();
        *reinterpret_cast<volatile int64_t*>(part.arrived) = 1;
      }
    }
  }
}

// (positions first .. n of the batch)
__global__ void __launch_bounds__(kBlock) touch_after_kernel(const int64_t* __restrict__ locs, int64_t first, int64_t n,
                                                             TouchMarks t, int32_t* __restrict__ after) {
  const uint32_t number = batch_number(t.batch);
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = first + warp * 32; base < n; base += nwarps * 32) {
    const int64_t i = base + lane;
    int64_t slot = i < n ? locs[i] : -1;
    if (slot >= t.capacity) slot = -1;
    const unsigned same = __match_any_sync(0xffffffffu, slot);
    if (slot < 0 || (same >> lane) != 1u) continue;
    uint32_t last[kWays];
    line_marks(t.marks, slot >> 3, number, last);
#pragma unroll
    for (int w = 0; w < kWays; ++w) {
      if (w == (int)(slot & 7) || !last[w] || last[w] > (uint32_t)(i + 1)) continue;
      // position p of this slot counts when p + 1 > last[w]: lanes from last[w] - base on
      const int64_t from = (int64_t)last[w] - base;
      const unsigned later = from <= 0 ? same : (from >= 32 ? 0u : same & ~((1u << from) - 1u));
      if (later) atomicAdd(after + (slot & ~(int64_t)7) + w, __popc(later));
    }
  }
}

__global__ void __launch_bounds__(kBlock) touch_apply_kernel(const int64_t* __restrict__ locs, int64_t first, int64_t n,
                                                             TouchMarks t, int32_t* __restrict__ after,
                                                             int32_t* __restrict__ line_hits, int32_t* __restrict__ lru,
                                                             unsigned long long* aged, unsigned long long lookup) {
  const uint32_t number = batch_number(t.batch);
  for (int64_t i = first + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t slot = locs[i];
    if (slot < 0 || slot >= t.capacity) continue;
    const int64_t line = slot >> 3;
    // the line is taken by the last hit of its lowest hit way
    if (t.marks[slot] != (((unsigned long long)number << 32) | (unsigned long long)(i + 1))) continue;
    uint32_t last[kWays];
    line_marks(t.marks, line, number, last);
    bool first = true;
#pragma unroll
    for (int w = 0; w < kWays; ++w)
      if (w < (int)(slot & 7) && last[w]) first = false;
    if (!first) continue;
    const int32_t total = line_hits[line];
    line_hits[line] = 0;
#pragma unroll
    for (int w = 0; w < kWays; ++w) {
      const int64_t x = line * kWays + w;
      if (last[w]) {
        lru[x] = after[x];
        after[x] = 0;
      } else {
        lru[x] += total;
      }
    }
  }
  if (batch_done(t.batch, number, gridDim.x) && aged) {  // (nullable: which batch of host ids this was)
    __threadfence();
    *reinterpret_cast<volatile unsigned long long*>(aged) = lookup;
  }
}

__global__ void aged_kernel(unsigned long long* aged, unsigned long long lookup) { *aged = lookup; }

// The same for large batches, sorted by slot: the marks are a line of memory and an atomic or two per hit.
__global__ void touch_keys_kernel(const int64_t* __restrict__ locs, int64_t n, int64_t capacity,
                                  uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t s = locs[i];
  keys[i] = (s >= 0 && s < capacity) ? (uint32_t)s : (uint32_t)capacity;
  vals[i] = (uint32_t)i;
}

__device__ __forceinline__ int64_t lower_bound_u32(const uint32_t* a, int64_t lo, int64_t hi,
                                                   uint32_t key) {
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// keys = hit slots sorted ascending (stable, so batch positions ascend inside a
// slot).  The thread at the head of each line's segment computes its counters.
__global__ void touch_sorted_kernel(const uint32_t* __restrict__ keys,
                                    const uint32_t* __restrict__ vals, int64_t n, int64_t capacity,
                                    int32_t* __restrict__ lru) {
  const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t key = keys[j];
  if ((int64_t)key >= capacity) return;  // misses sort last
  const uint32_t line = key >> 3;
  if (j > 0 && (keys[j - 1] >> 3) == line) return;
  // run boundaries of the 8 ways inside this line's segment
  int64_t rb[kWays + 1];
  rb[0] = j;
  // first position whose key belongs to a later line (or a miss)
  int64_t seg_hi = n;
  {
    // gallop to bound the binary search by the segment length, not by n
    int64_t step = 8;
    int64_t hi = j + 1;
    const uint32_t next = (line + 1) << 3;
    while (hi < n && keys[hi] < next) { hi = (hi + step < n) ? hi + step : n; step <<= 1; }
    seg_hi = lower_bound_u32(keys, j, hi, next);
  }
#pragma unroll
  for (int w = 1; w < kWays; ++w) rb[w] = lower_bound_u32(keys, rb[w - 1], seg_hi, (line << 3) + w);
  rb[kWays] = seg_hi;
  const int32_t total = (int32_t)(seg_hi - j);
#pragma unroll
  for (int w = 0; w < kWays; ++w) {
    int32_t* c = lru + (int64_t)line * kWays + w;
    if (rb[w + 1] == rb[w]) {
      *c += total;
    } else {
      const uint32_t last = vals[rb[w + 1] - 1];
      int32_t after = 0;
#pragma unroll
      for (int x = 0; x < kWays; ++x) {
        if (x == w || rb[x + 1] == rb[x]) continue;
        // positions in run x greater than `last`
        int64_t lo = rb[x], hi = rb[x + 1];
        while (lo < hi) {
          const int64_t mid = (lo + hi) >> 1;
          if (vals[mid] <= last) lo = mid + 1; else hi = mid;
        }
        after += (int32_t)(rb[x + 1] - lo);
      }
      *c = after;
    }
  }
}

// ---- LRU touch from runs -------------------------------------------------------
// The batch is given as runs of equal ids (each run = the sorted batch positions
// of one id, ascending), so "hits on the line after my last hit" is counted by
// binary search in the position lists of the other hit ways of the line, found through the marks.
__global__ void touch_runs_mark_kernel(RunsView v, TouchMarks marks) {
  begin_after_previous();
  const int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (u < v.runs()) marks.mark(v.slot_of_run(u), u);
}

__global__ void __launch_bounds__(kBlock) touch_runs_apply_kernel(RunsView v, TouchMarks t, int32_t* lru) {
  begin_after_previous();
  touch_runs(v, t, lru, blockIdx.x, gridDim.x);
}

// ---- reset -------------------------------------------------------------------
__global__ void reset_kernel(const int64_t* __restrict__ ids, int64_t n, int64_t lines,
                             int64_t* __restrict__ line_ids, int32_t* __restrict__ lru) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t id = ids[i];
  if (id < 0) return;
  const int64_t line = mod_nonneg(id, lines);
#pragma unroll
  for (int w = 0; w < kWays; ++w) {
    if (line_ids[line * kWays + w] == id) {
      line_ids[line * kWays + w] = -1;  // set_id(way, -1) also zeroes the counter
      lru[line * kWays + w] = 0;
      break;
    }
  }
}

// ---- enumerate / sorted view -------------------------------------------------
struct SlotValid {
  const int64_t* line_ids;
  __device__ bool operator()(int64_t slot) const { return line_ids[slot] != -1; }
};

__global__ void gather_ids_kernel(const int64_t* __restrict__ line_ids,
                                  const int64_t* __restrict__ slots, int64_t n,
                                  int64_t* __restrict__ ids_out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) ids_out[i] = line_ids[slots[i]];
}

__global__ void write_pairs_kernel(const int64_t* __restrict__ ids, const int64_t* __restrict__ slots,
                                   int64_t n, int64_t n_pad, longlong2* __restrict__ pairs) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n_pad) return;
  pairs[i] = i < n ? make_longlong2(ids[i], slots[i]) : make_longlong2(INT64_MAX, -1);
}

// level 1 samples the pairs with stride 8, higher levels sample the level below
// with stride 16
__global__ void build_level1_kernel(const longlong2* __restrict__ pairs, int64_t len,
                                    int64_t len_pad, int64_t* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= len_pad) return;
  out[i] = i < len ? pairs[i * kLeafFan].x : INT64_MAX;
}

__global__ void build_level_kernel(const int64_t* __restrict__ below, int64_t len, int64_t len_pad,
                                   int64_t* __restrict__ out) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= len_pad) return;
  out[i] = i < len ? below[i * kNodeFan] : INT64_MAX;
}

__global__ void count_valid_kernel(const int64_t* __restrict__ line_ids, int64_t n,
                                   unsigned long long* __restrict__ out) {
  unsigned long long c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    c += line_ids[i] != -1;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if (lane_id() == 0 && c) atomicAdd(out, c);
}

int grid_for(int64_t n, int block = kBlock) {
  int64_t g = ceil_div(n, block);
  if (g < 1) g = 1;
  return (int)g;
}

int grid_capped(int64_t n, int block = kBlock) {
  int64_t g = ceil_div(n, block);
  const int64_t cap = (int64_t)sm_count() * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

// the rest of the ageing by the marked positions first .. n; lookup: the batch of host ids that is complete then
static int age_marked(hb_index* h, const int64_t* locs, int64_t first, int64_t n, cudaStream_t st,
                      unsigned long long lookup = 0) {
  const int grid = grid_capped(n - first);
  const TouchMarks t = index_touch_marks(h);
  HB_LAUNCH(touch_after_kernel, grid, kBlock, 0, st, locs, first, n, t, h->after);
  HB_LAUNCH(touch_apply_kernel, grid, kBlock, 0, st, locs, first, n, t, h->after, h->line_hits, h->lru,
            lookup ? h->aged : nullptr, lookup);
  return HB_OK;
}

// (a number of its own for every stream there ever was: handles come back)
static bool eager_stream(cudaStream_t st, unsigned long long* id) {
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &c) == cudaSuccess && c == cudaStreamCaptureStatusNone &&
      cudaStreamGetId(st, id) == cudaSuccess)
    return true;
  cudaGetLastError();
  return false;
}

int IndexTurn::on(cudaStream_t st, bool goes_on) {
  st_ = st;
  used_ = eager_stream(st, &id_);
  if (!used_) return HB_OK;
  if (h_->was_changed && id_ != h_->changed_on) {
    if (h_->unrecorded) {
      int dev = h_->device;
      HB_CUDA(cudaGetDevice(&dev));
      if (dev != h_->device) HB_CUDA(cudaSetDevice(h_->device));
      const cudaError_t e = cudaEventRecord(h_->changed, cudaStreamLegacy);
      if (dev != h_->device) HB_CUDA(cudaSetDevice(dev));
      HB_CUDA(e);
      h_->unrecorded = false;
    }
    HB_CUDA(cudaStreamWaitEvent(st, h_->changed, 0));
  }
  if (goes_on || h_->open_first == h_->open_end) return HB_OK;
  const int64_t first = h_->open_first;
  h_->open_first = h_->open_end;
  return age_marked(h_, h_->open_locs, first, h_->open_end, st);
}

IndexTurn::~IndexTurn() {
  if (!used_) return;
  // (an event costs the call a microsecond or two)
  h_->unrecorded = st_ == nullptr || st_ == cudaStreamLegacy;
  if (!h_->unrecorded && cudaEventRecord(h_->changed, st_) != cudaSuccess) {
    cudaGetLastError();  // (the launches of the call have failed too)
    return;
  }
  h_->changed_on = id_;
  h_->was_changed = true;
}

int index_touch_apply(hb_index* h, const RunsView& v, cudaStream_t st) {
  HB_LAUNCH_NEXT(touch_runs_apply_kernel, grid_capped(v.max_runs), kBlock, 0, st, v, index_touch_marks(h), h->lru);
  return HB_OK;
}

// Where sets may get more ids than this on average, putting lists in order takes longer than the sort.
constexpr int64_t kListedPerSet = 16;
// One launch of the sort beats the launches of the lists up to here (add() of host ids: 2,000 33 us against
// 32, 4,000 39 against 40, 6,000 49 against 42, 8,000 57 against 45).
constexpr int64_t kAddSortMax = 8 * (int64_t)kClusterT;

// Positions that age through marks; more are sorted by slot (us, marks / sorted, skewed and uniform slots of a
// cache of 4,000,000: 65,536 26 / 74 and 23 / 67, 524,288 74 / 91 and 63 / 80, 1,048,576 131 / 106 and 112 / 94,
// 2,000,000 216 / 150 and 181 / 136).
constexpr int64_t kTouchMarksMax = 3 << 18;

static size_t touch_sort_temp_bytes(int64_t n) {
  size_t bytes = 0;
  cub::DoubleBuffer<uint32_t> k(nullptr, nullptr), v(nullptr, nullptr);
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, k, v, (int)n, 0, 32, (cudaStream_t)0);
  return bytes;
}
static size_t touch_sort_bytes(int64_t n) {
  return 4 * align_up((size_t)n * sizeof(uint32_t), 256) + align_up(touch_sort_temp_bytes(n), 256) + 256;
}

static size_t add_workspace_bytes(int64_t n) {
  if (n <= 0) return 256;
  return align_up((size_t)n * 4, 256) + align_up((size_t)n * sizeof(uint2), 256) + sort_grid_bytes(n) + 1024;
}

size_t index_add_runs_bytes(int64_t n) { return add_workspace_bytes(n); }
bool index_add_runs_lists(const hb_index* h, int64_t n) { return n <= kListedPerSet * h->lines; }

int index_add_runs_sorted(hb_index* h, const AddEntries& e, void* ws, int64_t* locs, uint8_t* last_writer,
                          cudaStream_t st) {
  Carver cv(ws);
  uint2* sorted = cv.take<uint2>(e.n);
  int64_t* cut = cv.take<int64_t>(1);
  HB_LAUNCH(add_cut_kernel, 1, kBlock, 0, st, e, cut);
  h->sorted_stale = true;
  return sort_run(ListedSource{e.ids, e.n, e.n_dev, e.listed, cut, h->lines},
                  AddFinish{h->line_ids, h->lru, locs, last_writer, sorted, false}, e.n, cv.take<char>(0), st);
}

}  // namespace hb

using namespace hb;

extern "C" {

namespace {
// everything of an index except its lines: the sorted view's storage, the scratch word and what add and the
// ageing keep between kernels (13.5 bytes a slot; with the index, so that every call may be captured)
int alloc_derived(hb_index_t* h) {
  const int64_t cap = h->cache_size;
  // level capacities for a full index
  int64_t len = h->lines;  // level 1: one id per leaf block
  int64_t total = 0;
  for (int l = 1; l < kMaxLevels; ++l) {
    h->level_off[l] = total;
    h->level_cap[l] = len + kNodeFan;
    total += align_up(h->level_cap[l], 32);
    len = ceil_div(len, kNodeFan);
  }
  // one allocation for all of it: each costs an index some 0.1 to 1 ms, and again when it goes
  const size_t pairs_bytes = align_up((cap + kLeafFan) * sizeof(longlong2), 256);
  const size_t level_bytes = align_up(total * sizeof(int64_t), 256);
  const size_t batch_bytes = align_up((size_t)cap * 12 + (size_t)h->lines * 12 + 8 * sizeof(int32_t), 256);
  HB_CUDA(cudaMalloc(&h->batch_scratch, batch_bytes + pairs_bytes + level_bytes + 4 * sizeof(int64_t)));
  HB_CUDA(cudaMemsetAsync(h->batch_scratch, 0, batch_bytes, 0));
  h->marks = static_cast<unsigned long long*>(h->batch_scratch);
  h->heads = h->marks + cap;
  h->after = reinterpret_cast<int32_t*>(h->heads + h->lines);
  h->line_hits = h->after + cap;
  h->batch = h->line_hits + h->lines;
  char* rest = static_cast<char*>(h->batch_scratch) + batch_bytes;
  h->pairs = reinterpret_cast<longlong2*>(rest);
  h->level_store = reinterpret_cast<int64_t*>(rest + pairs_bytes);
  h->scratch_count = reinterpret_cast<int64_t*>(rest + pairs_bytes + level_bytes);
  device_error_word();  // (allocated on first use)
  HB_CUDA(cudaEventCreateWithFlags(&h->changed, cudaEventDisableTiming));
  h->aged = reinterpret_cast<unsigned long long*>(h->lru + cap);
  h->sorted_stale = true;
  h->view.line_ids = h->line_ids;
  h->view.lines = h->lines;
  h->view.pairs = h->pairs;
  h->view.top = 0;
  return HB_OK;
}

struct IndexIpcHandle {
  int64_t cache_size;
  int64_t lines;
  cudaIpcMemHandle_t line_ids;
  cudaIpcMemHandle_t lru;
};
}  // namespace

int hb_index_create(int64_t cache_size, hb_index_t** out) {
  HB_CHECK_ARG(out != nullptr, "hb_index_create: out is null");
  HB_CHECK_ARG(cache_size > 0, "hb_index_create: cache_size must be positive");
  const int64_t lines = ceil_div(cache_size, kWays);
  HB_CHECK_ARG(lines <= ((int64_t)1 << 28), "hb_index_create: at most 2^31 slots are supported");
  hb_index_t* h = new hb_index_t();  // (all members zero)
  HB_CUDA(cudaGetDevice(&h->device));
  h->lines = lines;
  h->cache_size = lines * kWays;
  const int64_t cap = h->cache_size;
  HB_CUDA(cudaMalloc(&h->line_ids, cap * sizeof(int64_t)));
  // (and the word of the lookups, which an opener reads)
  HB_CUDA(cudaMalloc(&h->lru, cap * sizeof(int32_t) + sizeof(unsigned long long)));
  HB_CUDA(cudaMemsetAsync(h->lru + cap, 0, sizeof(unsigned long long), 0));
  int rc = alloc_derived(h);
  if (rc != HB_OK) return rc;
  HB_LAUNCH(fill_i64_kernel, grid_capped(cap), kBlock, 0, 0, h->line_ids, cap, (int64_t)-1);
  HB_LAUNCH(fill_i32_kernel, grid_capped(cap), kBlock, 0, 0, h->lru, cap, 0);
  HB_CUDA(cudaStreamSynchronize(0));
  *out = h;
  return HB_OK;
}

// An index shared between the processes of one box, as the reference shares its index through
// a named POSIX segment (SACacheIndex(name, create, ...), src/cache/cache.h:145-167): the
// creating process exports a handle, another process opens it and works on the SAME lines
// (ids and LRU counters) in the creator's HBM.  As in the reference nothing orders the two
// processes' calls: callers do (its test does with barriers, test/test_cache.py:20-55).
size_t hb_index_handle_bytes(void) { return sizeof(IndexIpcHandle); }

int hb_index_export_handle(hb_index_t* h, void* handle_out) {
  HB_CHECK_ARG(h && handle_out, "hb_index_export_handle: null argument");
  HB_CHECK_ARG(!h->opened, "hb_index_export_handle: only the creating process exports");
  IndexIpcHandle x;
  memset(&x, 0, sizeof(x));
  x.cache_size = h->cache_size;
  x.lines = h->lines;
  HB_CUDA(cudaIpcGetMemHandle(&x.line_ids, h->line_ids));
  HB_CUDA(cudaIpcGetMemHandle(&x.lru, h->lru));
  memcpy(handle_out, &x, sizeof(x));
  return HB_OK;
}

int hb_index_open(const void* handle, hb_index_t** out) {
  HB_CHECK_ARG(handle && out, "hb_index_open: null argument");
  IndexIpcHandle x;
  memcpy(&x, handle, sizeof(x));
  HB_CHECK_ARG(x.lines > 0 && x.cache_size == x.lines * kWays, "hb_index_open: not an index handle");
  hb_index_t* h = new hb_index_t();  // (all members zero)
  HB_CUDA(cudaGetDevice(&h->device));
  h->lines = x.lines;
  h->cache_size = x.cache_size;
  h->shared = true;
  h->opened = true;
  void* p = nullptr;
  HB_CUDA(cudaIpcOpenMemHandle(&p, x.line_ids, cudaIpcMemLazyEnablePeerAccess));
  h->line_ids = static_cast<int64_t*>(p);
  HB_CUDA(cudaIpcOpenMemHandle(&p, x.lru, cudaIpcMemLazyEnablePeerAccess));
  h->lru = static_cast<int32_t*>(p);
  int rc = alloc_derived(h);
  if (rc != HB_OK) return rc;
  HB_CUDA(cudaStreamSynchronize(0));
  *out = h;
  return HB_OK;
}

int hb_index_destroy(hb_index_t* h) {
  if (!h) return HB_OK;
  if (h->opened) {
    cudaIpcCloseMemHandle(h->line_ids);
    cudaIpcCloseMemHandle(h->lru);
  } else {
    cudaFree(h->line_ids);
    cudaFree(h->lru);
  }
  cudaFree(h->batch_scratch);  // (the sorted view's storage too)
  if (h->changed) cudaEventDestroy(h->changed);
  delete h;
  return HB_OK;
}

int64_t hb_index_size(const hb_index_t* h) { return h ? h->cache_size : -1; }
int64_t hb_index_capacity(const hb_index_t* h) { return h ? h->lines * kWays : -1; }
// bytes of one reference cache line: 8 int64 ids + 8 int32 counters
int64_t hb_index_space(const hb_index_t* h) { return h ? h->lines * 96 : -1; }
int64_t hb_index_lines(const hb_index_t* h) { return h ? h->lines : -1; }

int hb_index_valid_entries(hb_index_t* h, int64_t* out_host, hb_stream_t stream) {
  HB_CHECK_ARG(h && out_host, "hb_index_valid_entries: null argument");
  cudaStream_t st = (cudaStream_t)stream;
  HB_CUDA(cudaMemsetAsync(h->scratch_count, 0, sizeof(int64_t), st));
  HB_LAUNCH(count_valid_kernel, grid_capped(h->cache_size), kBlock, 0, st, h->line_ids,
            h->cache_size, (unsigned long long*)h->scratch_count);
  HB_CUDA(cudaMemcpyAsync(out_host, h->scratch_count, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  HB_CUDA(cudaStreamSynchronize(st));
  return HB_OK;
}

size_t hb_index_add_workspace_bytes(int64_t n) { return add_workspace_bytes(n); }
size_t hb_index_touch_lru_workspace_bytes(int64_t n) { return n > kTouchMarksMax ? touch_sort_bytes(n) : 256; }

int hb_index_add(hb_index_t* h, const int64_t* ids, int64_t n, int64_t* locs,
                 uint8_t* last_writer, void* workspace, size_t workspace_bytes,
                 hb_stream_t stream) {
  HB_CHECK_ARG(h && (n == 0 || (ids && locs)), "hb_index_add: null argument");
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31), "hb_index_add: n out of range");
  if (n == 0) return HB_OK;
  if (workspace_bytes < add_workspace_bytes(n) || !workspace) {
    set_error("hb_index_add: workspace of %zu bytes needed, %zu given", add_workspace_bytes(n), workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  int rc = turn.on(st);
  if (rc != HB_OK) return rc;
  Carver cv(workspace);
  h->sorted_stale = true;
  uint32_t* next = cv.take<uint32_t>(n);
  uint2* sorted = cv.take<uint2>(n);
  void* sort_ws = cv.take<char>(0);
  if (n > kAddSortMax && n <= kListedPerSet * h->lines) {
    HB_LAUNCH_NEXT(add_push_kernel, grid_for(n), kBlock, 0, st, ids, n, index_add_lists(h, next), locs, last_writer);
    AddEntries e;
    memset(&e, 0, sizeof(e));
    e.ids = ids;
    e.n = n;
    HB_LAUNCH_NEXT(add_walk_kernel, grid_capped(n), kBlock, 0, st, e, index_add_state(h, next, locs, last_writer));
    return sort_run(SetSource<true>{ids, n, h->lines, h->heads, h->batch + 2},
                    AddFinish{h->line_ids, h->lru, locs, last_writer, sorted, false}, n, sort_ws, st);
  }
  // (a cluster that holds more than one entry per thread leaves the walk to the whole GPU)
  AddFinish fin{h->line_ids, h->lru, locs, last_writer, sorted, n > kAddSortMax && n <= kSortClusterMax};
  rc = sort_run(SetSource<false>{ids, n, h->lines, nullptr, nullptr}, fin, n, sort_ws, st);
  if (rc != HB_OK || !fin.walk_later) return rc;
  HB_LAUNCH(add_sorted_walk_kernel, grid_for(n), kBlock, 0, st, ids, (int)n, fin);
  return HB_OK;
}

}  // extern "C"

// lookup of `ids` into locs (or the slots there, ids null: 64 bits only), first pass of the ageing
template <typename WORD>
static int touch_mark(hb_index* h, const WORD* ids, int64_t* locs, int64_t n, int mode, const HostPart<WORD>& part,
                      cudaStream_t st) {
  if (ids && mode == HB_LOOKUP_SORTED && h->sorted_stale) {
    const int rc = hb_index_build_sorted(h, st);
    if (rc != HB_OK) return rc;
  }
  const int grid = grid_capped(n);
  const TouchMarks t = index_touch_marks(h);
  if constexpr (sizeof(WORD) == sizeof(int64_t)) {
    if (!ids) {
      HB_LAUNCH((touch_mark_kernel<HB_LOOKUP_SETASSOC, false, WORD>), grid, kBlock, 0, st, h->view, ids, locs, n, t,
                h->line_hits, part);
      return HB_OK;
    }
  }
  if (mode == HB_LOOKUP_SORTED)
    HB_LAUNCH((touch_mark_kernel<HB_LOOKUP_SORTED, true, WORD>), grid, kBlock, 0, st, h->view, ids, locs, n, t, h->line_hits,
              part);
  else
    HB_LAUNCH((touch_mark_kernel<HB_LOOKUP_SETASSOC, true, WORD>), grid, kBlock, 0, st, h->view, ids, locs, n, t, h->line_hits,
              part);
  return HB_OK;
}

extern "C" {

// (workspace large enough for it)
static int touch_sorted(hb_index* h, const int64_t* locs, int64_t n, void* workspace, cudaStream_t st) {
  Carver cv(workspace);
  uint32_t* k0 = cv.take<uint32_t>(n);
  uint32_t* k1 = cv.take<uint32_t>(n);
  uint32_t* v0 = cv.take<uint32_t>(n);
  uint32_t* v1 = cv.take<uint32_t>(n);
  size_t temp_bytes = touch_sort_temp_bytes(n);
  void* temp = cv.take<char>(temp_bytes);
  HB_LAUNCH(touch_keys_kernel, grid_for(n), kBlock, 0, st, locs, n, h->cache_size, k0, v0);
  cub::DoubleBuffer<uint32_t> keys(k0, k1), vals(v0, v1);
  int bits = 1;
  while (bits < 32 && ((int64_t)1 << bits) < h->cache_size + 1) ++bits;
  HB_CUDA(cub::DeviceRadixSort::SortPairs(temp, temp_bytes, keys, vals, (int)n, 0, bits, st));
  count_library_launches(3);
  HB_LAUNCH(touch_sorted_kernel, grid_for(n), kBlock, 0, st, keys.Current(), vals.Current(), n, h->cache_size, h->lru);
  return HB_OK;
}

int hb_index_touch_lru(hb_index_t* h, const int64_t* locs, int64_t n, void* workspace, size_t workspace_bytes,
                       hb_stream_t stream) {
  HB_CHECK_ARG(h && (n == 0 || locs), "hb_index_touch_lru: null argument");
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31), "hb_index_touch_lru: n out of range");
  if (n == 0) return HB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  int rc = turn.on(st);
  if (rc == HB_OK && n > kTouchMarksMax && workspace && workspace_bytes >= touch_sort_bytes(n))
    return touch_sorted(h, locs, n, workspace, st);
  if (rc == HB_OK)
    rc = touch_mark<int64_t>(h, nullptr, const_cast<int64_t*>(locs), n, HB_LOOKUP_SETASSOC, {0, nullptr, nullptr}, st);
  return rc != HB_OK ? rc : age_marked(h, locs, 0, n, st);
}

static int check_lookup(hb_index_t* h, const void* ids, int64_t n, const int64_t* locs, int64_t first, int mode) {
  HB_CHECK_ARG(h && first >= 0 && (n == 0 || (ids && locs)), "hb_index_lookup_touch: null argument");
  HB_CHECK_ARG(mode == HB_LOOKUP_SETASSOC || mode == HB_LOOKUP_SORTED, "hb_index_lookup_touch: unknown mode %d", mode);
  HB_CHECK_ARG(n >= 0 && first + n < ((int64_t)1 << 31), "hb_index_lookup_touch: n out of range");
  return HB_OK;
}

int hb_index_lookup_touch(hb_index_t* h, const int64_t* ids, int64_t n, int64_t* locs, int mode,
                          hb_stream_t stream) {
  int rc = check_lookup(h, ids, n, locs, 0, mode);
  if (rc != HB_OK || n == 0) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  rc = turn.on(st);
  if (rc == HB_OK) rc = touch_mark<int64_t>(h, ids, locs, n, mode, {0, nullptr, nullptr}, st);
  return rc != HB_OK ? rc : age_marked(h, locs, 0, n, st);
}

}  // extern "C"

template <typename WORD>
static int lookup_touch_part(hb_index_t* h, const WORD* ids, int64_t n, int64_t* locs, int64_t first, WORD* host_locs,
                             int64_t* arrived, int mode, cudaStream_t st) {
  int rc = check_lookup(h, ids, n, locs, first, mode);
  if (rc != HB_OK || n == 0) return rc;
  IndexTurn turn(h);
  const bool next = h->open_locs == locs && h->open_end == first && h->open_first < first;
  rc = turn.on(st, next);
  if (rc == HB_OK) rc = touch_mark<WORD>(h, ids, locs + first, n, mode, {first, host_locs, arrived}, st);
  if (rc != HB_OK) return rc;
  h->open_locs = locs;
  if (!next) h->open_first = first;
  h->open_end = first + n;
  return HB_OK;
}

extern "C" {

int hb_index_lookup_touch_part(hb_index_t* h, const int64_t* ids, int64_t n, int64_t* locs, int64_t first,
                               int64_t* host_locs, int64_t* arrived, int mode, hb_stream_t stream) {
  return lookup_touch_part<int64_t>(h, ids, n, locs, first, host_locs, arrived, mode, (cudaStream_t)stream);
}

int hb_index_lookup_touch_part32(hb_index_t* h, const int32_t* ids, int64_t n, int64_t* locs, int64_t first,
                                 int32_t* host_locs, int64_t* arrived, int mode, hb_stream_t stream) {
  // (slots fit: hb_index_create makes no more than 2^31)
  return lookup_touch_part<int32_t>(h, ids, n, locs, first, host_locs, arrived, mode, (cudaStream_t)stream);
}

int hb_index_lookup_touch_end(hb_index_t* h, const int64_t* locs, int64_t n, hb_stream_t stream) {
  HB_CHECK_ARG(h && locs && n > 0, "hb_index_lookup_touch: no part of the batch was looked up");
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  int rc = turn.on(st, true);  // (also behind a call that has found the parts and aged by them: locs may be freed)
  if (rc != HB_OK) return rc;
  const int64_t first = h->open_first;
  const unsigned long long lookup = h->opened ? 0 : ++h->lookups;  // (the word is the creator's)
  if (h->open_locs == locs && h->open_end == n && first < n) {
    h->open_first = n;
    return age_marked(h, locs, first, n, st, lookup);
  }
  if (lookup) HB_LAUNCH(aged_kernel, 1, 1, 0, st, h->aged, lookup);
  return HB_OK;
}

uint64_t hb_index_lookups(const hb_index_t* h) { return h ? h->lookups : 0; }

int hb_index_wait_lookups(hb_index_t* h, uint64_t lookups, hb_stream_t stream) {
  HB_CHECK_ARG(h, "hb_index_wait_lookups: null index");
  cudaStream_t st = (cudaStream_t)stream;
  const auto until = std::chrono::steady_clock::now() + std::chrono::seconds(30);
  for (;;) {
    unsigned long long done = 0;
    HB_CUDA(cudaMemcpyAsync(&done, h->aged, sizeof(done), cudaMemcpyDeviceToHost, st));
    HB_CUDA(cudaStreamSynchronize(st));
    if (done >= lookups) return HB_OK;
    if (std::chrono::steady_clock::now() > until) break;
    std::this_thread::sleep_for(std::chrono::microseconds(50));
  }
  set_error("hb_index_wait_lookups: the creator's lookups do not end");
  return HB_ERR_TIMEOUT;
}

int hb_index_touch_lru_runs(hb_index_t* h, const int64_t* locs, const uint32_t* perm,
                            const int64_t* run_start, int64_t max_runs, const int64_t* num_runs,
                            int64_t n, const int64_t* n_dev, int locs_kind, hb_stream_t stream) {
  HB_CHECK_ARG(h && (n == 0 || locs), "hb_index_touch_lru_runs: null argument");
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31) && max_runs >= 0 && max_runs <= n,
               "hb_index_touch_lru_runs: sizes out of range");
  HB_CHECK_ARG(!(perm && !run_start), "hb_index_touch_lru_runs: a position list needs run starts");
  HB_CHECK_ARG(locs_kind >= 0 && locs_kind <= 2, "hb_index_touch_lru_runs: locs_kind is 0, 1 or 2");
  if (n == 0 || max_runs == 0) return HB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  const int rc = turn.on(st);
  if (rc != HB_OK) return rc;
  RunsView v{locs, perm, run_start, num_runs, n_dev, max_runs, n, locs_kind};
  HB_LAUNCH_NEXT(touch_runs_mark_kernel, grid_for(max_runs), kBlock, 0, st, v, index_touch_marks(h));
  return index_touch_apply(h, v, st);
}

int hb_index_lookup(hb_index_t* h, const int64_t* ids, int64_t n, int64_t* locs, uint8_t* found,
                    int mode, hb_stream_t stream) {
  HB_CHECK_ARG(h && (n == 0 || ids), "hb_index_lookup: null argument");
  HB_CHECK_ARG(mode == HB_LOOKUP_SETASSOC || mode == HB_LOOKUP_SORTED,
               "hb_index_lookup: unknown mode %d", mode);
  HB_CHECK_ARG(n >= 0, "hb_index_lookup: negative n");
  if (n == 0) return HB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const int grid = grid_capped(n);
  if (mode == HB_LOOKUP_SORTED) {
    if (h->sorted_stale) {
      int rc = hb_index_build_sorted(h, stream);
      if (rc != HB_OK) return rc;
    }
    HB_LAUNCH(lookup_kernel<HB_LOOKUP_SORTED>, grid, kBlock, 0, st, h->view, ids, n, locs, found);
  } else {
    HB_LAUNCH(lookup_kernel<HB_LOOKUP_SETASSOC>, grid, kBlock, 0, st, h->view, ids, n, locs, found);
  }
  return HB_OK;
}

int hb_index_reset(hb_index_t* h, const int64_t* ids, int64_t n, hb_stream_t stream) {
  HB_CHECK_ARG(h && (n == 0 || ids), "hb_index_reset: null argument");
  if (n <= 0) return HB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  const int rc = turn.on(st);
  if (rc != HB_OK) return rc;
  HB_LAUNCH(reset_kernel, grid_for(n), kBlock, 0, st, ids, n, h->lines, h->line_ids, h->lru);
  h->sorted_stale = true;
  return HB_OK;
}

// Select the valid slots (ascending) into a fresh device buffer; returns their
// count on the host.  Setup path: allocates and synchronises.
static int select_valid_slots(hb_index_t* h, cudaStream_t st, int64_t** slots_out,
                              int64_t* count_host) {
  const int64_t cap = h->cache_size;
  int64_t* slots = nullptr;
  HB_CUDA(cudaMalloc(&slots, cap * sizeof(int64_t)));
  cub::CountingInputIterator<int64_t> it(0);
  SlotValid pred{h->line_ids};
  size_t temp_bytes = 0;
  cub::DeviceSelect::If(nullptr, temp_bytes, it, slots, h->scratch_count, cap, pred, st);
  void* temp = nullptr;
  HB_CUDA(cudaMalloc(&temp, temp_bytes ? temp_bytes : 1));
  cudaError_t e = cub::DeviceSelect::If(temp, temp_bytes, it, slots, h->scratch_count, cap, pred, st);
  count_library_launches(2);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(count_host, h->scratch_count, sizeof(int64_t), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  cudaFree(temp);
  if (e != cudaSuccess) {
    cudaFree(slots);
    set_error("select_valid_slots: %s", cudaGetErrorString(e));
    return HB_ERR_CUDA;
  }
  *slots_out = slots;
  return HB_OK;
}

int hb_index_getall(hb_index_t* h, int64_t* ids_out, int64_t* locs_out, int64_t len,
                    int64_t* n_written_host, hb_stream_t stream) {
  HB_CHECK_ARG(h && len >= 0, "hb_index_getall: bad argument");
  HB_CHECK_ARG(len == 0 || (ids_out && locs_out), "hb_index_getall: null output");
  cudaStream_t st = (cudaStream_t)stream;
  int64_t* slots = nullptr;
  int64_t valid = 0;
  int rc = select_valid_slots(h, st, &slots, &valid);
  if (rc != HB_OK) return rc;
  const int64_t m = valid < len ? valid : len;
  cudaError_t e = cudaSuccess;
  if (m > 0) {
    e = cudaMemcpyAsync(locs_out, slots, m * sizeof(int64_t), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) {
      gather_ids_kernel<<<grid_for(m), kBlock, 0, st>>>(h->line_ids, slots, m, ids_out);
      count_launch();
      e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  }
  cudaFree(slots);
  if (e != cudaSuccess) {
    set_error("hb_index_getall: %s", cudaGetErrorString(e));
    return HB_ERR_CUDA;
  }
  if (n_written_host) *n_written_host = m;
  return HB_OK;
}

int hb_index_build_sorted(hb_index_t* h, hb_stream_t stream) {
  HB_CHECK_ARG(h, "hb_index_build_sorted: null index");
  cudaStream_t st = (cudaStream_t)stream;
  int64_t* slots = nullptr;
  int64_t valid = 0;
  int rc = select_valid_slots(h, st, &slots, &valid);
  if (rc != HB_OK) return rc;
  IndexView& v = h->view;
  v.line_ids = h->line_ids;
  v.lines = h->lines;
  v.pairs = h->pairs;
  for (int l = 0; l < kMaxLevels; ++l) { v.level[l] = nullptr; v.level_len[l] = 0; }
  v.top = 0;
  cudaError_t e = cudaSuccess;
  int64_t *ids = nullptr, *ids_sorted = nullptr, *slots_sorted = nullptr;
  void* temp = nullptr;
  if (valid > 0) {
    do {
      if ((e = cudaMalloc(&ids, valid * sizeof(int64_t))) != cudaSuccess) break;
      if ((e = cudaMalloc(&ids_sorted, valid * sizeof(int64_t))) != cudaSuccess) break;
      if ((e = cudaMalloc(&slots_sorted, valid * sizeof(int64_t))) != cudaSuccess) break;
      gather_ids_kernel<<<grid_for(valid), kBlock, 0, st>>>(h->line_ids, slots, valid, ids);
      count_launch();
      size_t temp_bytes = 0;
      cub::DeviceRadixSort::SortPairs(nullptr, temp_bytes, ids, ids_sorted, slots, slots_sorted,
                                      (int)valid, 0, 64, st);
      if ((e = cudaMalloc(&temp, temp_bytes ? temp_bytes : 1)) != cudaSuccess) break;
      if ((e = cub::DeviceRadixSort::SortPairs(temp, temp_bytes, ids, ids_sorted, slots,
                                               slots_sorted, (int)valid, 0, 64, st)) != cudaSuccess)
        break;
      count_library_launches(9);
      const int64_t n_pad = align_up(valid, kLeafFan);
      write_pairs_kernel<<<grid_for(n_pad), kBlock, 0, st>>>(ids_sorted, slots_sorted, valid, n_pad,
                                                             h->pairs);
      count_launch();
      v.level_len[0] = (int32_t)valid;
      int64_t len = n_pad / kLeafFan;
      for (int l = 1; l < kMaxLevels; ++l) {
        int64_t* out = h->level_store + h->level_off[l];
        const int64_t len_pad = align_up(len, kNodeFan);
        if (l == 1)
          build_level1_kernel<<<grid_for(len_pad), kBlock, 0, st>>>(h->pairs, len, len_pad, out);
        else
          build_level_kernel<<<grid_for(len_pad), kBlock, 0, st>>>(
              h->level_store + h->level_off[l - 1], len, len_pad, out);
        count_launch();
        v.level[l] = out;
        v.level_len[l] = (int32_t)len;
        if (len <= kTopMax) { v.top = l; break; }
        len = ceil_div(len, kNodeFan);
      }
      if ((e = cudaGetLastError()) != cudaSuccess) break;
      e = cudaStreamSynchronize(st);
    } while (0);
  }
  cudaFree(slots);
  cudaFree(ids);
  cudaFree(ids_sorted);
  cudaFree(slots_sorted);
  cudaFree(temp);
  if (e != cudaSuccess) {
    set_error("hb_index_build_sorted: %s", cudaGetErrorString(e));
    return HB_ERR_CUDA;
  }
  h->sorted_stale = h->shared;  // a shared index may change under this process
  return HB_OK;
}

int hb_index_export(hb_index_t* h, int64_t* line_ids, int32_t* lru, hb_stream_t stream) {
  HB_CHECK_ARG(h, "hb_index_export: null index");
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  const int rc = turn.on(st);
  if (rc != HB_OK) return rc;
  if (line_ids)
    HB_CUDA(cudaMemcpyAsync(line_ids, h->line_ids, h->cache_size * sizeof(int64_t),
                            cudaMemcpyDefault, st));
  if (lru)
    HB_CUDA(cudaMemcpyAsync(lru, h->lru, h->cache_size * sizeof(int32_t), cudaMemcpyDefault, st));
  HB_CUDA(cudaStreamSynchronize(st));
  return HB_OK;
}

int hb_index_import(hb_index_t* h, const int64_t* line_ids, const int32_t* lru,
                    hb_stream_t stream) {
  HB_CHECK_ARG(h, "hb_index_import: null index");
  cudaStream_t st = (cudaStream_t)stream;
  IndexTurn turn(h);
  const int rc = turn.on(st);
  if (rc != HB_OK) return rc;
  if (line_ids)
    HB_CUDA(cudaMemcpyAsync(h->line_ids, line_ids, h->cache_size * sizeof(int64_t),
                            cudaMemcpyDefault, st));
  if (lru)
    HB_CUDA(cudaMemcpyAsync(h->lru, lru, h->cache_size * sizeof(int32_t), cudaMemcpyDefault, st));
  HB_CUDA(cudaStreamSynchronize(st));
  h->sorted_stale = true;
  return HB_OK;
}

}  // extern "C"
