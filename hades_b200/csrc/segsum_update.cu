// Aggregation of duplicate gradients and the sparse optimiser's row update in one pass: what
// SparseAdam.update does with ids that repeat (python/EmbCache/sparse_optim.py:608-681: unique_grads,
// then state and table rows) without writing the merged rows and reading them back, and without
// the launches and the unique count between the two.
#include "segsum.cuh"

using namespace hb;

namespace {

int segsum_update(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim, int mean,
                  const hb_optim_t* opt, void* workspace, size_t workspace_bytes, bool zeroed, cudaStream_t st) {
  HB_CHECK_ARG(runs != nullptr && opt != nullptr && dim > 0, "hb_segsum_update_f32: bad argument");
  const int64_t n = runs->n;
  HB_CHECK_ARG(n == 0 || (grads && runs->perm && runs->head && runs->base8 && runs->run_start && runs->uniq_ids),
               "hb_segsum_update_f32: null argument");
  HB_CHECK_ARG(opt->kind == HB_OPT_ADAM || opt->kind == HB_OPT_ADAGRAD, "hb_segsum_update_f32: unknown optimiser");
  HB_CHECK_ARG(opt->emb && opt->s0 && (opt->kind != HB_OPT_ADAM || (opt->s1 && opt->step)),
               "hb_segsum_update_f32: incomplete optimiser description");
  HB_CHECK_ARG(opt->emb_elem_bytes == 4 || opt->emb_elem_bytes == 2,
               "hb_segsum_update_f32: embedding must be fp32 (4) or fp16 (2)");
  HB_CHECK_ARG(opt->rows > 0 && opt->id_stride > 0, "hb_segsum_update_f32: bad sizes");
  if (opt->rows >= ((int64_t)1 << 30)) {
    set_error("hb_segsum_update_f32: shards of 2^30 rows and more are not updated in one pass");
    return HB_ERR_UNSUPPORTED;
  }
  if (n == 0) return HB_OK;
  const uintptr_t bits = (uintptr_t)grads | (uintptr_t)opt->emb | (uintptr_t)opt->s0 | (uintptr_t)opt->s1;
  const bool vec4 = dim % 4 == 0 && (bits & 15) == 0;
  if (dim > seg_tile(vec4)) {
    // a row's step counter would be advanced once per pass over its columns
    set_error("hb_segsum_update_f32: rows of %lld columns are not updated in one pass", (long long)dim);
    return HB_ERR_UNSUPPORTED;
  }
  SegPlan s = seg_plan(workspace, n, dim);
  if (!workspace || workspace_bytes < s.total) {
    set_error("hb_segsum_update_f32: workspace of %zu bytes needed, %zu given", s.total, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  SegArgs a = seg_args(runs, grads, cnt_in, dim, mean, s);
  a.cols = (int)dim;
  if (!zeroed) HB_CUDA(cudaMemsetAsync(s.done, 0, (size_t)s.max_ctas * sizeof(unsigned), st));
  if (opt->kind == HB_OPT_ADAM) return seg_dispatch(a, update_rows<true, false>(runs, opt), vec4, st);
  return seg_dispatch(a, update_rows<false, false>(runs, opt), vec4, st);
}

}  // namespace

extern "C" {

int hb_segsum_update_f32(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim, int mean,
                         const hb_optim_t* opt, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  return segsum_update(runs, grads, cnt_in, dim, mean, opt, workspace, workspace_bytes, false, (cudaStream_t)stream);
}

int hb_unique_update_f32(const int64_t* ids, const float* grads, const int64_t* cnt_in, int64_t n, const int64_t* n_dev,
                         const int64_t* seg_counts, int64_t seg_cap, int64_t dim, int id_bits, int mean,
                         const hb_optim_t* opt, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31) && dim > 0, "hb_unique_update_f32: bad sizes");
  const size_t runs_bytes = align_up(hb_runs_workspace_bytes(n), 256);
  if (!workspace || workspace_bytes < runs_bytes + hb_segsum_runs_workspace_bytes(n, dim)) {
    set_error("hb_unique_update_f32: workspace of %zu bytes needed, %zu given",
              runs_bytes + hb_segsum_runs_workspace_bytes(n, dim), workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  char* seg_ws = static_cast<char*>(workspace) + runs_bytes;
  const SegPlan s = seg_plan(seg_ws, n, dim);
  hb_runs_t runs;
  int rc = runs_build(ids, n, n_dev, seg_counts, seg_cap, id_bits, nullptr, 0, nullptr, nullptr, nullptr, nullptr,
                      s.done, s.max_ctas, workspace, runs_bytes, &runs, (cudaStream_t)stream);
  if (rc != HB_OK) return rc;
  return segsum_update(&runs, grads, cnt_in, dim, mean, opt, seg_ws, workspace_bytes - runs_bytes, true,
                       (cudaStream_t)stream);
}

}  // extern "C"
