// The grouping of a batch of ids into runs of equal ids (hb_runs_t): what the sort of a
// step leaves behind, shared by the forward fetch (each distinct id is looked up and read
// once), the LRU ageing, the list of cache misses and the backward aggregation.
#pragma once

#include "common.cuh"

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

// hb_runs_build (without the sorted ids of the entries, which nothing here reads: runs_keys); zero: words that the launch after it needs at zero (set by the sort's own launch)
int runs_build(const int64_t* ids, int64_t n, const int64_t* n_dev, const int64_t* seg_counts, int64_t seg_cap,
               int id_bits, const int8_t* class_table, int64_t table_len, int64_t* const* class_ids_out,
               int64_t* class_counts_out, int64_t* uniq_ids_out, int64_t* num_unique_out, unsigned* zero,
               int64_t zero_words, void* workspace, size_t workspace_bytes, hb_runs_t* runs_out, cudaStream_t st);

// The sorted id of every entry (hb_runs_t.keys) of runs built in a plan that has room for them.
int runs_keys(const int64_t* seg_counts, int id_bits, void* workspace, hb_runs_t* runs, cudaStream_t st);

struct Maintain;
// The rows of a batch to its positions (run_src: where every run's row lies, bit 0 = a cache row), the
// index brought up to date in the same launch.
int runs_expand_maintain(const hb_runs_t* runs, const unsigned long long* run_src, const int64_t* run_slots,
                         const void* cache_rows, const void* table, int64_t row_bytes, void* out_rows, int64_t* locs,
                         uint8_t* found, const Maintain& duty, cudaStream_t st);

#ifdef __CUDACC__
__device__ __forceinline__ int64_t runs_valid_entries(const hb_runs_t& r) {
  if (!r.n_dev) return r.n;
  const int64_t d = *r.n_dev;
  return d < r.n ? (d > 0 ? d : 0) : r.n;
}
#endif

}  // namespace hb
