// Device-resident cache index: state layout and the lookup device functions
// shared by the stand-alone lookup kernels and the fused lookup+fetch kernels.
//
// State of record (what add/reset/touch_lru mutate), structure-of-arrays form of
// the reference's 96-byte cache_line (src/cache/cache_line.h:7-11):
//   line_ids[lines*8]  int64   -1 = empty        one 64-byte line per set
//   lru     [lines*8]  int32   access counters
// Derived, read-only "sorted view" for HB_LOOKUP_SORTED:
//   pairs[]            (id, slot) sorted by id, padded to 8 with (INT64_MAX,-1)
//   level[1..top][]    level[1] = id of every 8th pair, level[k+1] = every 16th
//                      id of level[k]; each padded with INT64_MAX so that a
//                      16-key block read never leaves the array.  The top level
//                      (<= kTopMax ids) is staged in shared memory by each CTA.
#pragma once

#include <mutex>

#include "common.cuh"

#ifdef __CUDACC__
#define HB_DEV __device__ __forceinline__
#else
#define HB_DEV inline
#endif

namespace hb {

constexpr int kWays = HB_WAYS;
constexpr int kMaxLevels = 8;     // enough for 2^40 ids
constexpr int kTopMax = 2048;     // ids of the top level held in shared memory
constexpr int kLeafFan = 8;       // pairs per leaf block (128 bytes)
constexpr int kNodeFan = 16;      // ids per inner block (128 bytes)

struct IndexView {
  const int64_t* line_ids;
  int64_t lines;
  // sorted view
  const longlong2* pairs;
  const int64_t* level[kMaxLevels];  // level[0] unused
  int32_t level_len[kMaxLevels];     // valid ids per level (level[0]: pairs)
  int32_t top;                       // index of the top level (>= 1), 0 if empty
};

}  // namespace hb

struct hb_index {
  int device;
  int64_t cache_size;  // capacity = lines * 8 (reference: _init_cache, cache.h:47)
  int64_t lines;
  int64_t* line_ids;   // [lines*8]
  int32_t* lru;        // [lines*8]
  // sorted view
  bool sorted_stale;
  longlong2* pairs;            // [round_up(capacity, 8) + 8]
  int64_t* level_store;        // one allocation, levels carved from it
  int64_t level_off[hb::kMaxLevels];
  int64_t level_cap[hb::kMaxLevels];
  int64_t* scratch_count;      // device int64[4] for small reductions
  // scratch of add and of the LRU ageing, one allocation made with the index; entries are valid when their
  // batch number is that of the batch at work, so nothing is cleared between batches (32 bits:
  // 2^31 batches per index).  The batch numbers live on the device: a captured graph advances them.
  void* batch_scratch;
  unsigned long long* marks;    // [capacity] (batch << 32) | 1 + last position / run that hit the slot
  int32_t* after;               // [capacity] hits on the line after the slot's last; zero between calls
  int32_t* line_hits;           // [lines] zero between calls
  unsigned long long* heads;    // [lines] (batch << 32) | 1 + entry: list of the batch's ids of a set
  int32_t* batch;               // [8] touch: batch, blocks done; add: batch, blocks done, batch with long lists
  hb::IndexView view;
  // An index over another process's lines (hb_index_open): the sorted view is this process's
  // own and is rebuilt before every use, because the owner may have changed the lines since.
  // (The owner itself rebuilds after its own changes; after a change by the other process it
  // calls hb_index_build_sorted.)
  bool shared;
  bool opened;  // line_ids / lru are mappings of another process's memory
  // Calls that change lines or counters take turns (IndexTurn): they share the scratch above.
  std::mutex turn;
  cudaEvent_t changed;            // behind the last such call
  unsigned long long changed_on;  // the id of its stream
  bool was_changed;
  bool unrecorded;                // ... on the default stream, which stays: recorded when another one has to wait
  unsigned long long lookups;     // batches of host ids so far
  unsigned long long* aged;       // behind lru on the device: the last of them whose ageing is done
  // a batch of host ids of which some parts are looked up: positions that wait for their ageing
  const int64_t* open_locs;
  int64_t open_first, open_end;
};

#ifdef __CUDACC__
namespace hb {

// ---- set-associative probe ---------------------------------------------------
// The warp resolves 32 queries (lane l owns id_l).  Groups of 8 lanes read one
// 64-byte line per step; 4 queries per step, 8 steps.  Returns the slot of this
// lane's own id (or -1).
__device__ __forceinline__ int64_t warp_lookup_setassoc(const IndexView& v, int64_t id) {
  const int lane = lane_id();
  const int sub = lane & 7;
  const int grp = lane >> 3;
  const bool valid = id >= 0;
  const int64_t line = valid ? mod_nonneg(id, v.lines) : -1;
  int64_t keys[8];
  int64_t qid[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int q = r * 4 + grp;
    const int64_t lq = __shfl_sync(0xffffffffu, line, q);
    qid[r] = __shfl_sync(0xffffffffu, id, q);
    keys[r] = lq >= 0 ? v.line_ids[lq * kWays + sub] : (int64_t)-1;
  }
  int64_t slot = -1;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const unsigned b = __ballot_sync(0xffffffffu, qid[r] >= 0 && keys[r] == qid[r]);
    if ((lane >> 2) == r) {
      const unsigned mine = (b >> ((lane & 3) * 8)) & 0xffu;
      // the reference's find() returns the FIRST matching way (cache_line.h:49-55)
      if (mine) slot = line * kWays + (__ffs(mine) - 1);
    }
  }
  return slot;
}

// A lane probes the line of its own id: all lines are on their way at once, and it takes half the registers, so that more
// warps of an SM wait for theirs (a step of 282,624 ids 403 -> 397.5 us, of 2,000,000 742.5 -> 740, of 65,536 107.8 ->
// 106.8; lookup and fetch of 65,536 rows of 512 bytes 13.1 -> 11.0, of 1,500,000 of 64 bytes 58.2 -> 51.0).
__device__ __forceinline__ int64_t lane_lookup(const int64_t* line_ids, int64_t lines, int64_t id) {
  int64_t slot = -1;
  if (id >= 0) {
    const int64_t line = mod_nonneg(id, lines);
    const longlong2* p = reinterpret_cast<const longlong2*>(line_ids + line * kWays);
    longlong2 k[kWays / 2];
#pragma unroll
    for (int w = 0; w < kWays / 2; ++w) k[w] = p[w];
#pragma unroll
    for (int w = kWays / 2 - 1; w >= 0; --w) {  // the FIRST way that matches (cache_line.h:49-55)
      if (k[w].y == id) slot = line * kWays + 2 * w + 1;
      if (k[w].x == id) slot = line * kWays + 2 * w;
    }
  }
  return slot;
}

// ---- sorted-view search --------------------------------------------------------
// top level must already be in shared memory (stage_top_level).
__device__ __forceinline__ void stage_top_level(const IndexView& v, int64_t* smem_top) {
  if (v.top == 0) return;
  const int n = v.level_len[v.top];
  for (int i = threadIdx.x; i < n; i += blockDim.x) smem_top[i] = v.level[v.top][i];
}

__device__ __forceinline__ int64_t warp_lookup_sorted(const IndexView& v, const int64_t* smem_top,
                                                      int64_t id) {
  const int lane = lane_id();
  const int sub = lane & 7;
  const int grp = lane >> 3;
  if (v.top == 0) return -1;
  // per-lane upper_bound over the shared-memory top level
  int64_t t = -1;
  if (id >= 0) {
    int lo = 0, hi = v.level_len[v.top];
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (smem_top[mid] <= id) lo = mid + 1; else hi = mid;
    }
    t = lo - 1;
  }
  // inner levels: 16 ids per block, two per lane of an 8-lane group
  for (int l = v.top - 1; l >= 1; --l) {
    const longlong2* lv = reinterpret_cast<const longlong2*>(v.level[l]);
    longlong2 k[8];
    int64_t qid[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int q = r * 4 + grp;
      const int64_t tq = __shfl_sync(0xffffffffu, t, q);
      qid[r] = __shfl_sync(0xffffffffu, id, q);
      k[r] = tq >= 0 ? lv[tq * (kNodeFan / 2) + sub] : make_longlong2(INT64_MAX, INT64_MAX);
    }
    int64_t nt = t;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const unsigned b0 = __ballot_sync(0xffffffffu, k[r].x <= qid[r]);
      const unsigned b1 = __ballot_sync(0xffffffffu, k[r].y <= qid[r]);
      if ((lane >> 2) == r && t >= 0) {
        const int sh = (lane & 3) * 8;
        const int c = __popc((b0 >> sh) & 0xffu) + __popc((b1 >> sh) & 0xffu);
        nt = t * kNodeFan + c - 1;  // c >= 1: the block's first id is the parent id
      }
    }
    t = nt;
  }
  // leaf: 8 (id, slot) pairs per block, one per lane of the group
  longlong2 p[8];
  int64_t qid[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const int q = r * 4 + grp;
    const int64_t tq = __shfl_sync(0xffffffffu, t, q);
    qid[r] = __shfl_sync(0xffffffffu, id, q);
    p[r] = tq >= 0 ? v.pairs[tq * kLeafFan + sub] : make_longlong2(INT64_MAX, -1);
  }
  int64_t slot = -1;
#pragma unroll
  for (int r = 0; r < 8; ++r) {
    const unsigned b = __ballot_sync(0xffffffffu, p[r].x == qid[r] && qid[r] >= 0);
    // owner lane of query (r, g) is lane r*4+g; it takes the slot from the
    // matching lane of group g
    const int g_owner = lane & 3;
    const unsigned mine = (b >> (g_owner * 8)) & 0xffu;
    const int src = mine ? g_owner * 8 + (__ffs(mine) - 1) : 0;
    const int64_t s = __shfl_sync(0xffffffffu, p[r].y, src);
    if ((lane >> 2) == r && mine) slot = s;
  }
  return slot;
}

template <int MODE>
__device__ __forceinline__ int64_t warp_lookup(const IndexView& v, const int64_t* smem_top,
                                               int64_t id) {
  if (MODE == HB_LOOKUP_SORTED) return warp_lookup_sorted(v, smem_top, id);
  return warp_lookup_setassoc(v, id);
}

}  // namespace hb
#endif  // __CUDACC__

namespace hb {

#ifdef __CUDACC__
// One batch number for all blocks of a kernel, advanced by the block that finishes last (every block
// has read it by then): counter[0] batches so far, counter[1] blocks done.
__device__ __forceinline__ uint32_t batch_number(const int32_t* counter) { return (uint32_t)*counter + 1u; }
// True in one thread of that block.
__device__ __forceinline__ bool batch_done(int32_t* counter, uint32_t number, int blocks) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(reinterpret_cast<unsigned*>(counter + 1), 1u) == (unsigned)blocks - 1u) {
      counter[1] = 0;
      counter[0] = (int32_t)number;
      return true;
    }
  }
  return false;
}
#endif

// A batch grouped in runs of equal ids, as the LRU ageing sees it.
struct RunsView {
  const int64_t* locs;       // slot of every batch position (or of every sorted entry, see below)
  const uint32_t* perm;      // nullable: position list of the runs (identity when null)
  const int64_t* run_start;  // nullable: run u = [run_start[u], run_start[u+1]) (run u = {u} when null)
  const int64_t* num_runs;   // nullable device count
  const int64_t* n_dev;      // nullable device count of positions
  int64_t max_runs;
  int64_t n;
  int locs_kind;             // locs holds a slot per batch position (0), per sorted entry (1), per run (2)
  HB_DEV int64_t slot_of_run(int64_t u) const {
    if (locs_kind == 2) return locs[u];
    const int64_t j = start(u);
    return locs[locs_kind == 1 ? j : pos(j)];
  }
  HB_DEV int64_t positions() const {
    if (!n_dev) return n;
    const int64_t d = *n_dev;
    return d < n ? (d > 0 ? d : 0) : n;
  }
  HB_DEV int64_t runs() const {
    int64_t r = max_runs;
    if (num_runs && *num_runs < r) r = *num_runs;
    if (!run_start) { const int64_t p = positions(); if (p < r) r = p; }
    return r;
  }
  HB_DEV int64_t start(int64_t u) const { return run_start ? run_start[u] : u; }
  HB_DEV int64_t end(int64_t u, int64_t nruns, int64_t npos) const {
    return (u + 1 < nruns) ? start(u + 1) : npos;
  }
  HB_DEV int64_t pos(int64_t j) const { return perm ? (int64_t)perm[j] : j; }
};

// What a kernel that looks ids up leaves for the ageing of their hits (index_touch_apply).
struct TouchMarks {
  unsigned long long* marks;
  int32_t* batch;
  int64_t capacity;
#ifdef __CUDACC__
  __device__ __forceinline__ void mark(int64_t slot, int64_t run) const {
    if (slot >= 0 && slot < capacity)
      marks[slot] = ((unsigned long long)batch_number(batch) << 32) | (unsigned long long)(run + 1);
  }
#endif
};

// What a kernel that finds new ids leaves for their insertion (index_add_walk): entry i at the front
// of the list of its set.
struct AddLists {
  unsigned long long* heads;
  int32_t* batch;
  uint32_t* next;   // [n] 1 + the entry behind this one, 0 = none
  int64_t lines;
#ifdef __CUDACC__
  __device__ __forceinline__ void push(int64_t id, int64_t i) const {
    const unsigned long long b = (unsigned long long)batch_number(batch) << 32;
    const unsigned long long was = atomicExch(heads + mod_nonneg(id, lines), b | (unsigned long long)(i + 1));
    next[i] = (was >> 32) == (b >> 32) ? (uint32_t)was : 0u;
  }
#endif
};

// Entries that were put on the lists: all n, or (a batch whose lookups missed) those at work[] with
// at most `cap` of them taken, the first ones.
struct AddEntries {
  const int64_t* ids;            // [n] id of an entry
  int64_t n;
  const int64_t* n_dev;          // nullable: entries, on the device
  const uint8_t* listed;         // nullable [n]: entry is on a list (else: non-negative ids are)
  const int32_t* chunk_listed;   // nullable: listed entries of 32 at a time
  const unsigned long long* total;  // their number
  int64_t cap;
};

// The turn of a call that changes an index: from one thread at a time (the kernels of a call are enqueued
// together), and behind the last such call where that one went to another stream.  Streams inside a capture are
// ordered by whoever replays the graph.
class IndexTurn {
 public:
  explicit IndexTurn(hb_index* h) : h_(h), lock_(h->turn) {}
  ~IndexTurn();
  // The stream of the launches to come, before the first of them.  A batch that another thread looks up in
  // parts is aged by its parts so far (one hit after the other: cut in two it ages the same), unless this call
  // is its next.
  int on(cudaStream_t st, bool goes_on = false);

 private:
  hb_index* h_;
  std::lock_guard<std::mutex> lock_;
  cudaStream_t st_ = nullptr;
  unsigned long long id_ = 0;
  bool used_ = false;
};

inline TouchMarks index_touch_marks(const hb_index* h) { return TouchMarks{h->marks, h->batch, h->cache_size}; }
int index_touch_apply(hb_index* h, const RunsView& v, cudaStream_t st);
inline AddLists index_add_lists(const hb_index* h, uint32_t* next) { return AddLists{h->heads, h->batch + 2, next, h->lines}; }
// add() of the distinct ids of a batch that `listed` names: slots and "last writer of its slot" flags
// for them; beyond the cap -1 / 0.  Where index_add_runs_lists says so through the lists of their sets
// (AddLists, Maintain), else sorted by set.
size_t index_add_runs_bytes(int64_t n);
bool index_add_runs_lists(const hb_index* h, int64_t n);
int index_add_runs_sorted(hb_index* h, const AddEntries& e, void* ws, int64_t* locs, uint8_t* last_writer,
                          cudaStream_t st);

}  // namespace hb
