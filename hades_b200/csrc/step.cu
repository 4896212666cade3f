// One trainer's step on one GPU in two calls (hb_step_forward / hb_step_backward).
//
//   forward   sort | per distinct id: probe, place its row is read from, mark of a hit for the ageing,
//             a missed cold id onto the list of its set | rows to the batch positions, meanwhile LRU
//             ageing and the listed ids into the index | rows of the inserted ids into the cache
//   backward  per distinct cold id: probe, staging entry, mark | gradients summed, hot rows updated,
//             cold rows staged, meanwhile LRU ageing
//
// What bounds it: at 2,000 ids nothing but launches (composed from separate calls the same work took
// 33 launches and 450 us of host time for 160 us of kernels); at 2,000,000 ids HBM.
#include "index.cuh"
#include "launch.cuh"
#include "maintain.cuh"
#include "runs.cuh"
#include "segsum.cuh"
#include "staging.cuh"

struct hb_step {
  int device;
  cudaStream_t side;
  cudaEvent_t forked, fetched;
  bool side_busy;    // `fetched` has to be waited for
  hb_runs_t runs;    // of the last batch
  int64_t runs_n;    // 0: none
};

namespace hb {
int* device_error_word();  // runtime.cu

namespace {

constexpr int kBlock = 256;
constexpr int kCold = 2;
// Small batches update rows as their sums become complete (one launch); large ones write the sums and
// update in a second pass over the distinct ids: the sums then run at the speed of the copy, and the
// update has many rows in flight whatever the lengths of the runs.
// The line lies where the two cost the same for 128 columns (us a step with flushes, Adam, forward and backward called apart,
// at once / in a second pass: 50,000 ids of 16 columns 72.4 / 72.0, of 64 80.2 / 81.6, of 128 96.6 / 98.6, of 256 128.8 / 127.4;
// 75,000: 85.9 / 83.9, 100.8 / 97.8, 123.5 / 122.2, 165.0 / 160.9; 100,000: 96.3 / 93.9, 116.7 / 113.3, 139.0 / 133.2, 203.8 /
// 188.9; Adagrad 50,000 of 128 90.5 / 93.6, 75,000 116.5 / 116.4, 100,000 130.1 / 126.9).  By width it would lie lower: 65,000 of
// 16 76.2 / 74.5, for Adagrad 74.8 / 70.8, of 64 87.1 / 85.8 and 85.6 / 82.6, of 128 104.8 / 106.3 and 99.8 / 100.2, of 256 142.9 /
// 139.9 and 135.2 / 134.2; 20,000 of 64 63.6 / 65.3, of 256 78.1 / 84.7, of 16 for Adagrad 58.4 / 55.9.
// In a captured step, and in one call above the line, the fetch runs beside the sums.
constexpr int64_t kFuseMax = 70000;
constexpr int64_t kFewRows = 100000;
bool fuses_update(int64_t n) { return n <= kFuseMax; }

constexpr int kListedWords = 64;  // of the counter, which all warps add to: a line of its own

struct StepPlan {
  char* runs_ws;
  size_t runs_bytes;
  void* fetch_ws;        // hb_lookup_fetch_runs_workspace_bytes: run_src first
  size_t fetch_bytes;
  int64_t* run_slots;    // [n] slot of every run at the lookup
  int64_t* cold_slots;   // [n] slot of every cold run at the accumulate
  int64_t* new_slots;    // [n] slot a missed cold run was given
  uint8_t* on_list;      // [n] the run is a cold miss, to be inserted
  uint8_t* last_writer;  // [n]
  void* add_ws;          // index_add_runs_bytes: the lists' links first
  // what the sort's launch sets to zero
  unsigned* zero;
  int64_t zero_words;
  unsigned long long* listed;  // [1]
  int32_t* chunk_listed; // [n / 32 + 1]
  SegPlan seg;           // its arrival counters among the zeroed words
  float* sums;           // [n][dim], where the update is a launch of its own
  size_t total;
};

StepPlan step_plan(void* ws, int64_t n, int64_t dim) {
  StepPlan p;
  Carver cv(ws ? ws : (void*)256);
  const int64_t m = n > 0 ? n : 1;
  p.runs_bytes = make_runs_plan(nullptr, m, false).total;
  p.runs_ws = cv.take<char>(p.runs_bytes);
  p.fetch_bytes = hb_lookup_fetch_runs_workspace_bytes(m, 1, 0);
  p.fetch_ws = cv.take<char>(p.fetch_bytes);
  p.run_slots = cv.take<int64_t>(m);
  p.cold_slots = cv.take<int64_t>(m);
  p.new_slots = cv.take<int64_t>(m);
  p.on_list = cv.take<uint8_t>(m);
  p.last_writer = cv.take<uint8_t>(m);
  p.add_ws = cv.take<char>(index_add_runs_bytes(m));
  const SegPlan sizes = seg_plan(nullptr, m, dim);
  const int64_t chunks = m / 32 + 1;
  p.zero_words = kListedWords + chunks + sizes.max_ctas;
  p.zero = cv.take<unsigned>(p.zero_words);
  p.listed = reinterpret_cast<unsigned long long*>(p.zero);
  p.chunk_listed = reinterpret_cast<int32_t*>(p.zero + kListedWords);
  p.seg = seg_plan(cv.take<char>(sizes.total), m, dim);
  p.seg.done = p.zero + kListedWords + chunks;
  p.sums = cv.take<float>((size_t)m * dim);
  p.total = cv.used() + 256;
  return p;
}

// slot of a lane's own id (-1: none)
template <int MODE>
__device__ __forceinline__ int64_t step_lookup(const IndexView& v, const int64_t* s_top, int64_t id) {
  if constexpr (MODE == HB_LOOKUP_SORTED) return warp_lookup<MODE>(v, s_top, id);
  else return lane_lookup(v.line_ids, v.lines, id);
}
constexpr int step_lookup_blocks(int mode) { return mode == HB_LOOKUP_SORTED ? 2 : 6; }  // (an SM)

// The lookup of the runs in a launch of its own (resolve_run: as part of the sort's).
template <int MODE>
__global__ void __launch_bounds__(kBlock, step_lookup_blocks(MODE)) step_resolve_kernel(IndexView v, hb_runs_t r, RunsResolve a) {
  begin_after_previous();
  __shared__ int64_t s_top[MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  const int64_t U = *r.num_runs;
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u0 = warp * 32; u0 < U; u0 += nwarps * 32) {
    const int64_t u = u0 + lane;
    const int64_t id = u < U ? r.uniq_ids[u] : -1;
    const bool cold = u < U && r.dclass[u] == kCold;
    resolved_run<true>(a, u, u < U, id, cold, step_lookup<MODE>(v, s_top, id));
  }
}

int join_side(hb_step* s, cudaStream_t st) {
  if (s->side_busy) {
    HB_CUDA(cudaStreamWaitEvent(st, s->fetched, 0));
    s->side_busy = false;
  }
  return HB_OK;
}

struct ColdArgs {
  hb_staging_t s;
  const int32_t* thr_table;  // nullable
  int32_t default_thr;
  unsigned long long* dropped;  // nullable
  int64_t* slots;            // [runs]
  TouchMarks marks;
  int touch;
};

// The cold ids: slot now that this batch's misses are in the cache, staging entry (server.py:546-562 without the
// row), mark for the ageing.
template <int MODE>
__global__ void __launch_bounds__(kBlock, step_lookup_blocks(MODE)) step_cold_kernel(IndexView v, hb_runs_t r, ColdArgs a) {
  begin_after_previous();
  __shared__ int64_t s_top[MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  const int64_t U = *r.num_runs;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u0 = warp * 32; u0 < U; u0 += nwarps * 32) {
    const int64_t u = u0 + lane_id();
    const bool cold = u < U && r.dclass[u] == kCold;
    const int64_t id = cold ? r.uniq_ids[u] : -1;
    const int64_t slot = step_lookup<MODE>(v, s_top, id);
    if (slot >= 0) {
      a.s.idx[slot] = id;
      a.s.iter_threshold[slot] = a.thr_table ? a.thr_table[id] : a.default_thr;
      a.s.cnt[slot] += 1;
      if (a.touch) a.marks.mark(slot, u);
    }
    if (a.dropped) {
      const unsigned miss = __ballot_sync(0xffffffffu, cold && slot < 0);
      if (lane_id() == 0 && miss) atomicAdd(a.dropped, (unsigned long long)__popc(miss));
    }
    if (u < U) a.slots[u] = slot;
  }
}

// CTAs that run on an SM at once: 4 by 64 registers a thread, fewer where a lane holds more of a row.
constexpr int step_apply_ctas(bool adam, int vec, int vpl) {
  return vec * vpl <= (adam ? 4 : 8) ? 4 : 2;
}

// Summed gradients to where they belong: state and table rows of hot ids, staging rows of cold ones; then LRU
// ageing by the lookup that found the staging rows.  A warp takes 32 distinct ids a round, a lane each for what is worked
// out once per id, then G lanes per row.  Bound by HBM: rows read and written once.  As many warps as run at once, 32 an
// SM with one row in flight per lane group, walk the ids side by side in chunks of eight: no second, partly filled wave,
// and neighbouring rows of the table at one time (a stretch of its own for every warp: 10 us more).  A step of 282,624
// ids of 128 columns for Adam (85,000 hot, 76,000 cold) 411 -> 403 us, of 2,000,000 (88,000, 80,000) 751 -> 748; with 24
// warps and two rows in flight 427, with the ageing ahead of the rows 405.  (Two CTAs an SM where four fit, at other widths:
// 1,000,000 x 47 for Adam 559 us, with four 538, for Adagrad 513 and 492, 282,624 x 256 for Adagrad 310 and 301.)
template <bool ADAM, int VEC, int G, int VPL>
__global__ void __launch_bounds__(kBlock, step_apply_ctas(ADAM, VEC, VPL)) step_apply_kernel(hb_runs_t r, SegArgs a,
                                                                                           UpdateRows<ADAM, true> epi,
                                                                                           const float* sums) {
  begin_after_previous();
  const int row_blocks = (int)gridDim.x - epi.touch_blocks;
  if ((int)blockIdx.x >= row_blocks) {
    touch_runs(epi.touched, epi.marks, epi.lru, (int)blockIdx.x - row_blocks, epi.touch_blocks);
    return;
  }
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  apply_runs<ADAM, VEC, G, VPL>(epi, a, sums, 0, *r.num_runs, warp, ((int64_t)row_blocks * blockDim.x) >> 5);
}

template <bool ADAM, int VEC>
int launch_apply(const hb_runs_t& r, const SegArgs& a, const UpdateRows<ADAM, true>& epi, const float* sums,
                 cudaStream_t st) {
  const int vpr = a.cols / VEC;
#define HB_APPLY(G, VPL)                                                                                              \
  do {                                                                                                                \
    int64_t blocks = ceil_div(r.n, kBlock);                                                                           \
    const int64_t most = (int64_t)sm_count() * step_apply_ctas(ADAM, VEC, VPL); /* what runs at once */                \
    if (blocks > most) blocks = most;                                                                                 \
    HB_LAUNCH_NEXT((step_apply_kernel<ADAM, VEC, G, VPL>), (int)(blocks + epi.touch_blocks), kBlock, 0, st, r, a, epi, sums); \
  } while (0)
  if (vpr > 64) HB_APPLY(32, 4);
  else if (vpr > 32) HB_APPLY(32, 2);
  else if (vpr > 16) HB_APPLY(32, 1);
  else if (vpr > 8) HB_APPLY(16, 1);
  else if (vpr > 4) HB_APPLY(8, 1);
  else HB_APPLY(4, 1);
#undef HB_APPLY
  return HB_OK;
}

int grid_for_runs(int64_t n) {
  int64_t blocks = ceil_div(n, kBlock);
  const int64_t cap = (int64_t)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}

template <bool ADAM>
int update_step(hb_step* s, const hb_step_desc_t* d, const ColdArgs& c, SegArgs a, bool vec4, float* sums, bool fused,
                cudaStream_t st) {
  const hb_runs_t& r = s->runs;
  auto epi = update_rows<ADAM, true>(&r, &d->opt);
  epi.dclass = r.dclass;
  epi.staged = d->staging.grad;
  epi.slots = c.slots;
  if (d->touch_lru) {
    epi.touch_blocks = grid_for_runs(r.n);
    // the lookup of the accumulate: every distinct cold id once, in ascending order
    epi.touched = RunsView{c.slots, nullptr, nullptr, r.num_runs, r.num_runs, r.n, r.n, 2};
    epi.marks = c.marks;
    epi.lru = d->index->lru;
  }
  IndexTurn turn(d->index);
  auto look_up = [&](cudaStream_t on) -> int {
    const int rc = turn.on(on);
    if (rc != HB_OK) return rc;
    const IndexView& v = d->index->view;
    if (d->lookup_mode == HB_LOOKUP_SORTED)
      HB_LAUNCH_NEXT(step_cold_kernel<HB_LOOKUP_SORTED>, grid_for_runs(r.n), kBlock, 0, on, v, r, c);
    else
      HB_LAUNCH_NEXT(step_cold_kernel<HB_LOOKUP_SETASSOC>, grid_for_runs(r.n), kBlock, 0, on, v, r, c);
    return HB_OK;
  };
  epi.sums = sums;
  if (fused) {
    const int rc = look_up(st);
    return rc != HB_OK ? rc : seg_dispatch(a, epi, vec4, st);
  }
  // The sums need the sort only.  Beside them, once the cache holds the misses of this batch: where the cold ids are,
  // behind all that the caller has enqueued up to here (a fetch aside waits for less: for the forward call).
  HB_CUDA(cudaEventRecord(s->forked, st));
  HB_CUDA(cudaStreamWaitEvent(s->side, s->forked, 0));
  int rc = look_up(s->side);
  if (rc != HB_OK) return rc;
  HB_CUDA(cudaEventRecord(s->fetched, s->side));
  s->side_busy = true;
  StoreRows store;
  memset(&store, 0, sizeof(store));
  store.sums = sums;
  rc = seg_dispatch(a, store, vec4, st);
  // from here on the fetch of this batch must have read its rows
  if (rc == HB_OK) rc = join_side(s, st);
  if (rc == HB_OK) rc = turn.on(st);
  if (rc != HB_OK) return rc;
  return vec4 ? launch_apply<ADAM, 4>(r, a, epi, sums, st) : launch_apply<ADAM, 1>(r, a, epi, sums, st);
}

int check_desc(const hb_step_desc_t* d, const char* who) {
  if (!d || !d->index || !d->cache_rows || !d->table || !d->class_table || !d->staging.grad || d->row_bytes <= 0 ||
      d->dim <= 0 || d->table_rows <= 0 || d->class_len <= 0 || !d->opt.emb || !d->opt.s0) {
    set_error("%s: incomplete description", who);
    return HB_ERR_INVALID;
  }
  // (as the stand-alone updates refuse them: hb_sparse_adam, hb_sparse_adagrad)
  if (d->opt.kind != HB_OPT_ADAM && d->opt.kind != HB_OPT_ADAGRAD) {
    set_error("%s: unknown optimiser", who);
    return HB_ERR_INVALID;
  }
  if (d->opt.emb_elem_bytes != 4 && d->opt.emb_elem_bytes != 2) {
    set_error("%s: embedding must be fp32 (4) or fp16 (2)", who);
    return HB_ERR_INVALID;
  }
  if (d->opt.rows <= 0 || d->opt.id_stride <= 0 || (d->opt.kind == HB_OPT_ADAM && (!d->opt.s1 || !d->opt.step))) {
    set_error("%s: incomplete optimiser description", who);
    return HB_ERR_INVALID;
  }
  if (d->staging.slots != d->index->cache_size || d->staging.dim != d->dim) {
    set_error("%s: the staging table must have one slot per cache slot and rows of dim columns", who);
    return HB_ERR_INVALID;
  }
  return HB_OK;
}

bool vec4_ok(const hb_step_desc_t* d, const float* grads) {
  const uintptr_t bits = (uintptr_t)grads | (uintptr_t)d->opt.emb | (uintptr_t)d->opt.s0 | (uintptr_t)d->opt.s1 |
                         (uintptr_t)d->staging.grad;
  return d->dim % 4 == 0 && (bits & 15) == 0;
}

int build_runs(hb_step* s, const hb_step_desc_t* d, const StepPlan& p, const int64_t* ids, int64_t n,
               int64_t* counters, cudaStream_t st, const RunsResolve* resolve = nullptr) {
  const int rc = runs_build(ids, n, nullptr, nullptr, 0, d->id_bits, d->class_table, d->class_len, nullptr,
                            counters + 1, nullptr, counters, p.zero, p.zero_words, p.runs_ws, p.runs_bytes, &s->runs, st, resolve);
  s->runs_n = rc == HB_OK ? n : 0;
  return rc;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hb_step_create(hb_step_t** out) {
  HB_CHECK_ARG(out, "hb_step_create: out is null");
  hb_step* s = new hb_step();
  memset(s, 0, sizeof(*s));
  HB_CUDA(cudaGetDevice(&s->device));
  HB_CUDA(cudaStreamCreateWithFlags(&s->side, cudaStreamNonBlocking));
  HB_CUDA(cudaEventCreateWithFlags(&s->forked, cudaEventDisableTiming));
  HB_CUDA(cudaEventCreateWithFlags(&s->fetched, cudaEventDisableTiming));
  *out = s;
  return HB_OK;
}

int hb_step_destroy(hb_step_t* s) {
  if (!s) return HB_OK;
  cudaStreamDestroy(s->side);
  cudaEventDestroy(s->forked);
  cudaEventDestroy(s->fetched);
  delete s;
  return HB_OK;
}

size_t hb_step_workspace_bytes(int64_t n, int64_t dim) { return step_plan(nullptr, n, dim > 0 ? dim : 1).total; }

int hb_step_supported(const hb_step_desc_t* d) {
  if (check_desc(d, "hb_step_supported") != HB_OK) return 0;
  if (d->dim > seg_tile(vec4_ok(d, nullptr))) return 0;
  return d->opt.rows < ((int64_t)1 << 30) && d->staging.slots < ((int64_t)1 << 30);
}

int hb_step_join(hb_step_t* s, hb_stream_t stream) {
  HB_CHECK_ARG(s, "hb_step_join: null handle");
  return join_side(s, (cudaStream_t)stream);
}

int hb_step_forward(hb_step_t* s, const hb_step_desc_t* d, const int64_t* ids, int64_t n, void* out_rows,
                    int64_t* locs, uint8_t* found, int64_t* counters, int aside_allowed, void* workspace,
                    size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(s, "hb_step_forward: null handle");
  int rc = check_desc(d, "hb_step_forward");
  if (rc != HB_OK) return rc;
  HB_CHECK_ARG(n > 0 && n < ((int64_t)1 << 31), "hb_step_forward: n out of range");
  HB_CHECK_ARG(ids && out_rows && found && counters, "hb_step_forward: null argument");
  const StepPlan p = step_plan(workspace, n, d->dim);
  if (!workspace || workspace_bytes < p.total) {
    set_error("hb_step_forward: workspace of %zu bytes needed, %zu given", p.total, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  hb_index* h = d->index;
  rc = join_side(s, st);
  if (rc != HB_OK) return rc;
  if (d->lookup_mode == HB_LOOKUP_SORTED && h->sorted_stale) {
    rc = hb_index_build_sorted(h, stream);
    if (rc != HB_OK) return rc;
  }
  const bool lists_used = d->insert_misses && index_add_runs_lists(h, n);
  const RunsResolve a{h->line_ids, h->lines, (const char*)d->cache_rows, (const char*)d->table, d->table_rows, d->row_bytes,
                      static_cast<unsigned long long*>(p.fetch_ws), p.run_slots, d->insert_misses ? p.on_list : nullptr,
                      p.last_writer, p.chunk_listed, p.listed, lists_used, d->touch_lru, index_touch_marks(h),
                      index_add_lists(h, static_cast<uint32_t*>(p.add_ws)), device_error_word()};
  // aside: all of the fetch leaves the caller's stream, which goes on to the aggregation of the
  // same batch (it needs the sort only); both are bound by HBM, but not all the time
  const bool aside = aside_allowed && (stream_captures(st) || !fuses_update(n));
  const bool in_sort = !aside && n <= kResolvedMax && d->lookup_mode == HB_LOOKUP_SETASSOC;
  IndexTurn turn(h);
  if (in_sort) rc = turn.on(st);
  if (rc == HB_OK) rc = build_runs(s, d, p, ids, n, counters, st, in_sort ? &a : nullptr);
  if (rc != HB_OK) return rc;
  if (aside) {
    HB_CUDA(cudaEventRecord(s->forked, st));
    HB_CUDA(cudaStreamWaitEvent(s->side, s->forked, 0));
    st = s->side;
  }
  if (!in_sort) {
    rc = turn.on(st);
    if (rc != HB_OK) return rc;
    if (d->lookup_mode == HB_LOOKUP_SORTED)
      HB_LAUNCH_NEXT(step_resolve_kernel<HB_LOOKUP_SORTED>, grid_for_runs(n), kBlock, 0, st, h->view, s->runs, a);
    else
      HB_LAUNCH_NEXT(step_resolve_kernel<HB_LOOKUP_SETASSOC>, grid_for_runs(n), kBlock, 0, st, h->view, s->runs, a);
  }
  Maintain m;
  memset(&m, 0, sizeof(m));
  // Few rows: their blocks and those that bring the index up to date run at once, and what counts is the latter's chain
  // of reads: hits and misses to different blocks (2,000 ids 48.4 -> 48.0 us a step, 65,536 113.3 -> 112.6; 282,624 415.8 ->
  // 418.8).  Many: those blocks are spread among the rows', not ahead of them (282,624 415.8 -> 413, 2,000,000 750.4 ->
  // 745.4; 65,536 113.3 -> 114.2).  In between (us a step of 128 columns for Adam, apart / spread): 50,000 93.9 / 94.0, 65,000 105.0 /
  // 105.4, 80,000 123.5 / 122.3, 100,000 132.4 / 131.7, 120,000 145.8 / 145.0, 150,000 163.0 / 159.9; 16 to 256 columns alike.
  const bool few_rows = n <= kFewRows;
  if (lists_used) h->sorted_stale = true;  // (ageing leaves the ids where they are)
  if (d->touch_lru || lists_used) {
    m.v = RunsView{p.run_slots, s->runs.perm, s->runs.run_start, s->runs.num_runs, nullptr, n, n, 2};
    m.marks = a.marks;
    m.e = AddEntries{s->runs.uniq_ids, n, s->runs.num_runs, p.on_list, p.chunk_listed, p.listed, d->miss_cap};
    m.add = index_add_state(h, static_cast<uint32_t*>(p.add_ws), p.new_slots, p.last_writer);
    m.touch = d->touch_lru;
    m.insert = lists_used;
    m.apart = m.touch && m.insert && few_rows;
    m.blocks = grid_for_runs(n) * (m.apart ? 2 : 1);
    m.spread = !few_rows;
  }
  rc = runs_expand_maintain(&s->runs, a.run_src, p.run_slots, d->cache_rows, d->table, d->row_bytes, out_rows, locs,
                            found, m, st);
  if (rc != HB_OK) return rc;
  if (d->insert_misses) {
    if (!lists_used) {
      const AddEntries e{s->runs.uniq_ids, n, s->runs.num_runs, p.on_list, p.chunk_listed, p.listed, d->miss_cap};
      rc = index_add_runs_sorted(h, e, p.add_ws, p.new_slots, p.last_writer, st);
      if (rc != HB_OK) return rc;
    }
    rc = staging_insert_rows(&d->staging, d->table, s->runs.uniq_ids, n, s->runs.num_runs, d->cache_rows,
                             d->row_bytes, p.new_slots, p.last_writer, true, st);
    if (rc != HB_OK) return rc;
  }
  if (aside) {
    HB_CUDA(cudaEventRecord(s->fetched, st));
    s->side_busy = true;
  }
  return HB_OK;
}

int hb_step_backward(hb_step_t* s, const hb_step_desc_t* d, const int64_t* ids, int64_t n, const float* grads,
                     int64_t* counters, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(s, "hb_step_backward: null handle");
  int rc = check_desc(d, "hb_step_backward");
  if (rc != HB_OK) return rc;
  HB_CHECK_ARG(n > 0 && n < ((int64_t)1 << 31) && grads, "hb_step_backward: bad argument");
  HB_CHECK_ARG(ids ? counters != nullptr : s->runs_n == n, "hb_step_backward: not the batch of the last forward call");
  const StepPlan p = step_plan(workspace, n, d->dim);
  if (!workspace || workspace_bytes < p.total) {
    set_error("hb_step_backward: workspace of %zu bytes needed, %zu given", p.total, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  const bool vec4 = vec4_ok(d, grads);
  if (d->dim > seg_tile(vec4)) {
    set_error("hb_step_backward: rows of %lld columns are not updated in one pass", (long long)d->dim);
    return HB_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  hb_index* h = d->index;
  const bool fused = fuses_update(n) && !stream_captures(st);
  // A fetch that is still aside outside of the capture that this call belongs to (or inside one that it does not):
  // the join is refused, before the second stream takes work of this call.
  const bool apart = s->side_busy && stream_captures(st) != stream_captures(s->side);
  if (ids || fused || apart) {
    rc = join_side(s, st);
    if (rc != HB_OK) return rc;
  }
  if (ids) {
    rc = build_runs(s, d, p, ids, n, counters, st);
    s->runs_n = 0;  // the next forward pass is another batch
    if (rc != HB_OK) return rc;
  }
  if (d->lookup_mode == HB_LOOKUP_SORTED && h->sorted_stale) {
    rc = join_side(s, st);
    if (rc != HB_OK) return rc;
    rc = hb_index_build_sorted(h, stream);
    if (rc != HB_OK) return rc;
  }
  const TouchMarks marks = index_touch_marks(h);
  const ColdArgs c{d->staging, d->threshold_table, d->default_threshold, (unsigned long long*)d->dropped,
                   p.cold_slots, marks, d->touch_lru};
  SegArgs a = seg_args(&s->runs, grads, nullptr, d->dim, 0, p.seg);
  a.n_dev = nullptr;  // all entries: nothing to wait for
  a.cols = (int)d->dim;
  return d->opt.kind == HB_OPT_ADAM ? update_step<true>(s, d, c, a, vec4, p.sums, fused, st)
                                    : update_step<false>(s, d, c, a, vec4, p.sums, fused, st);
}

}  // extern "C"
