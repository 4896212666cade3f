// Hot-node local aggregation: sorted unique ids, per-id fp32 sum (or mean) of the
// duplicate-id gradient rows, per-id counts.  Replaces only_unique_grads /
// unique_grads (python/EmbCache/sparse_optim.py:132-157: torch.unique +
// index_add_).  The grouping comes from hb_runs_build (runs.cu; a step that fetched the same ids
// first hands its runs over instead), the sums from the kernel in segsum.cuh.
#include "segsum.cuh"

using namespace hb;

extern "C" {

size_t hb_segsum_runs_workspace_bytes(int64_t n, int64_t dim) { return seg_plan(nullptr, n, dim).total; }

int hb_segsum_runs_f32(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim,
                       int mean, float* sums, int64_t* counts, const hb_class_split_t* split,
                       void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  return segsum_runs(runs, grads, cnt_in, dim, mean, sums, counts, split, workspace, workspace_bytes, false, false,
                     (cudaStream_t)stream);
}

}  // extern "C"

int hb::segsum_runs(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim, int mean,
                    float* sums, int64_t* counts, const hb_class_split_t* split, void* workspace,
                    size_t workspace_bytes, bool zeroed, bool early, cudaStream_t st) {
  HB_CHECK_ARG(runs != nullptr && dim > 0, "hb_segsum_runs_f32: bad argument");
  const int64_t n = runs->n;
  HB_CHECK_ARG(n == 0 || (grads && runs->perm && runs->head && runs->base8 && runs->run_start && runs->num_runs),
               "hb_segsum_runs_f32: null argument");
  HB_CHECK_ARG(n == 0 || split || sums, "hb_segsum_runs_f32: null output");
  HB_CHECK_ARG(!split || n == 0 || (runs->dclass && runs->dpos),
               "hb_segsum_runs_f32: a split needs runs built with the class table");
  if (n == 0) return HB_OK;
  SegPlan s = seg_plan(workspace, n, dim);
  if (!workspace || workspace_bytes < s.total) {
    set_error("hb_segsum_runs_f32: workspace of %zu bytes needed, %zu given", s.total, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  uintptr_t align_bits = (uintptr_t)grads | (uintptr_t)sums;
  if (split)
    for (int c = 0; c < 3; ++c) align_bits |= (uintptr_t)split->out_rows[c];
  const bool vec4 = (dim % 4 == 0) && (align_bits & 15) == 0;
  SegArgs a = seg_args(runs, grads, cnt_in, dim, mean, s);
  a.early = early;
  StoreRows epi;
  epi.sums = sums;
  epi.dclass = split ? runs->dclass : nullptr;
  epi.dpos = runs->dpos;
  epi.counts = counts;
  for (int c = 0; c < 3; ++c) {
    epi.class_rows[c] = split ? split->out_rows[c] : nullptr;
    epi.class_counts[c] = split ? split->out_cnt[c] : nullptr;
  }
  if (!zeroed) HB_CUDA(cudaMemsetAsync(s.done, 0, (size_t)s.max_ctas * sizeof(unsigned), st));
  const int tile = seg_tile(vec4);
  for (int64_t col0 = 0; col0 < dim; col0 += tile) {
    a.col0 = col0;
    a.cols = (int)((dim - col0) < tile ? (dim - col0) : tile);
    const int rc = seg_dispatch(a, epi, vec4, st);
    if (rc != HB_OK) return rc;
  }
  return HB_OK;
}

extern "C" {

size_t hb_unique_segsum_workspace_bytes(int64_t n, int64_t dim) {
  return align_up(hb_runs_workspace_bytes(n), 256) + seg_plan(nullptr, n, dim).total;
}

int hb_unique_segsum_f32(const int64_t* ids, const float* grads, const int64_t* cnt_in, int64_t n,
                         const int64_t* n_dev, const int64_t* seg_counts, int64_t seg_cap,
                         int64_t dim, int id_bits, int mean,
                         int64_t* uniq_ids, float* sums,
                         int64_t* counts, int64_t* num_unique, hb_runs_t* runs_out,
                         const hb_class_split_t* split, void* workspace, size_t workspace_bytes,
                         hb_stream_t stream) {
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31) && dim > 0, "hb_unique_segsum_f32: bad sizes");
  HB_CHECK_ARG(num_unique != nullptr, "hb_unique_segsum_f32: num_unique is null");
  HB_CHECK_ARG(n == 0 || (ids && grads), "hb_unique_segsum_f32: null argument");
  HB_CHECK_ARG(n == 0 || split || (uniq_ids && sums), "hb_unique_segsum_f32: null output");
  HB_CHECK_ARG(!split || (split->table && split->class_counts && split->table_len > 0),
               "hb_unique_segsum_f32: a split needs the class table, its length and class_counts");
  const size_t runs_bytes = align_up(hb_runs_workspace_bytes(n), 256);
  if (!workspace || workspace_bytes < hb_unique_segsum_workspace_bytes(n, dim)) {
    set_error("hb_unique_segsum_f32: workspace of %zu bytes needed, %zu given",
              hb_unique_segsum_workspace_bytes(n, dim), workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  hb_runs_t runs;
  int64_t* cls_ids[3] = {split ? split->out_ids[0] : nullptr, split ? split->out_ids[1] : nullptr,
                         split ? split->out_ids[2] : nullptr};
  char* seg_ws = static_cast<char*>(workspace) + runs_bytes;
  const SegPlan s = seg_plan(seg_ws, n, dim);
  int rc = runs_build(ids, n, n_dev, seg_counts, seg_cap, id_bits, split ? split->table : nullptr,
                      split ? split->table_len : 0, split ? cls_ids : nullptr, split ? split->class_counts : nullptr,
                      uniq_ids, num_unique, s.done, s.max_ctas, workspace, runs_bytes, &runs, (cudaStream_t)stream);
  if (rc != HB_OK) return rc;
  if (runs_out) {
    rc = runs_keys(seg_counts, id_bits, workspace, &runs, (cudaStream_t)stream);
    if (rc != HB_OK) return rc;
    *runs_out = runs;
  }
  if (!n_dev && !seg_counts) runs.n_dev = nullptr;  // all entries: nothing to wait for
  return segsum_runs(&runs, grads, cnt_in, dim, mean, sums, counts, split, seg_ws, workspace_bytes - runs_bytes, true,
                     true, (cudaStream_t)stream);
}

}  // extern "C"
