// The grouping of a batch of ids into runs of equal ids (hb_runs_t): what the sort of a
// step leaves behind, shared by the forward fetch (each distinct id is looked up and read
// once), the LRU ageing, the list of cache misses and the backward aggregation.
#pragma once

#include "index.cuh"

namespace hb {

// carve of the workspace behind hb_runs_build
struct RunsPlan {
  uint32_t* perm;       // [m] positions
  void* sort_ws;
  int64_t* run_start;   // [m + 1]
  uint8_t* head;        // [m + 8]
  int64_t* n_valid;     // [1]
  int64_t* num_runs;    // [1]
  int64_t* class_counts;  // [4]
  int8_t* dclass;       // [m + 1]
  int32_t* dpos;        // [m + 1]
  int64_t* uniq;        // [m + 1]
  int32_t* base8;       // [m / 8 + 2]
  void* keys;           // [m] where hb_runs_t leaves the library: 4 or 8 bytes each
  size_t total;
};

RunsPlan make_runs_plan(void* ws, int64_t n, bool keys);

// What a step wants of every distinct id: the slot, where the row is read from, the mark of a hit for the ageing, a
// missed cold id onto the list of its set.
struct RunsResolve {
  const int64_t* line_ids;
  int64_t lines;
  const char* cache_rows;
  const char* table;
  int64_t table_rows;
  int64_t row_bytes;
  unsigned long long* run_src;  // where every run's row lies, bit 0 = a cache row
  int64_t* run_slots;
  uint8_t* on_list;       // nullable: misses are not inserted
  uint8_t* last_writer;
  int32_t* chunk_listed;  // per 32 runs
  unsigned long long* listed;  // zero before
  int push;               // ... onto the lists of their sets
  int touch;
  TouchMarks marks;
  AddLists lists;
  int* err;
};
// Up to here a thread of the sort has one run at most and looks it up where it writes it (us, sort and lookup: 2,000
// ids 13.4 + 4.0 and the boundary between them / 15.5; with 2.5 runs a thread, one after the other, 65,536 ids
// 34.1 + 5.3 / 43.6).
constexpr int64_t kResolvedMax = 8192;

// hb_runs_build (without the sorted ids of the entries, which nothing here reads: runs_keys).  zero: words that the
// sort's own launch sets to zero, for `resolve` or the launches after it.  resolve (up to kResolvedMax ids): done with
// every run, through the lines of the sets.
int runs_build(const int64_t* ids, int64_t n, const int64_t* n_dev, const int64_t* seg_counts, int64_t seg_cap,
               int id_bits, const int8_t* class_table, int64_t table_len, int64_t* const* class_ids_out,
               int64_t* class_counts_out, int64_t* uniq_ids_out, int64_t* num_unique_out, unsigned* zero,
               int64_t zero_words, void* workspace, size_t workspace_bytes, hb_runs_t* runs_out, cudaStream_t st,
               const RunsResolve* resolve = nullptr);

// The sorted id of every entry (hb_runs_t.keys) of runs built in a plan that has room for them.
int runs_keys(const int64_t* seg_counts, int id_bits, void* workspace, hb_runs_t* runs, cudaStream_t st);

struct Maintain;
// The rows of a batch to its positions (run_src: where every run's row lies, bit 0 = a cache row), the
// index brought up to date in the same launch.
int runs_expand_maintain(const hb_runs_t* runs, const unsigned long long* run_src, const int64_t* run_slots,
                         const void* cache_rows, const void* table, int64_t row_bytes, void* out_rows, int64_t* locs,
                         uint8_t* found, const Maintain& duty, cudaStream_t st);

#ifdef __CUDACC__
// Run u of a step and the slot its lookup found, one per lane (consecutive ones, the inactive lanes last); the
// whole warp calls it.  WHOLE: a warp's runs are a chunk of 32; else they lie in two, whose counts are zero before.
template <bool WHOLE>
__device__ __forceinline__ void resolved_run(const RunsResolve& a, int64_t u, bool valid, int64_t id, bool cold,
                                             int64_t slot) {
  if (a.on_list) {
    const bool missed = valid && cold && slot < 0;
    const unsigned m = __ballot_sync(0xffffffffu, missed);
    if (WHOLE) {
      if (lane_id() == 0) {
        a.chunk_listed[u >> 5] = __popc(m);
        if (m) atomicAdd(a.listed, (unsigned long long)__popc(m));
      }
    } else if (m) {
      const int64_t u0 = __shfl_sync(0xffffffffu, u, 0);
      const int cut = 32 - (int)(u0 & 31);
      const unsigned low = cut == 32 ? ~0u : (1u << cut) - 1u;
      if (lane_id() == 0) {
        if (m & low) atomicAdd(a.chunk_listed + (u0 >> 5), __popc(m & low));
        if (m & ~low) atomicAdd(a.chunk_listed + (u0 >> 5) + 1, __popc(m & ~low));
        atomicAdd(a.listed, (unsigned long long)__popc(m));
      }
    }
    if (missed && a.push) a.lists.push(id, u);
    if (valid) {
      a.on_list[u] = missed;
      a.last_writer[u] = 0;
    }
  }
  if (!valid) return;
  const char* src = nullptr;
  if (slot >= 0) src = a.cache_rows + slot * a.row_bytes;
  else if (id < a.table_rows) src = a.table + id * a.row_bytes;
  else atomicExch(a.err, HB_ERR_INVALID);  // no such row: the output rows of the run stay as they were
  a.run_src[u] = (unsigned long long)src | (slot >= 0 ? 1ull : 0ull);
  a.run_slots[u] = slot;
  if (a.touch) a.marks.mark(slot, u);
}

__device__ __forceinline__ void resolve_run(const RunsResolve& a, int64_t u, bool valid, int64_t id, bool cold) {
  resolved_run<false>(a, u, valid, id, cold, lane_lookup(a.line_ids, a.lines, valid ? id : -1));
}

__device__ __forceinline__ int64_t runs_valid_entries(const hb_runs_t& r) {
  if (!r.n_dev) return r.n;
  const int64_t d = *r.n_dev;
  return d < r.n ? (d > 0 ? d : 0) : r.n;
}
#endif

}  // namespace hb
