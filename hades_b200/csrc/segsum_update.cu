// Aggregation of duplicate gradients and the sparse optimiser's row update in one call: what
// SparseAdam.update does with ids that repeat (python/EmbCache/sparse_optim.py:608-681: unique_grads,
// then state and table rows), without the host reading the unique count between the two.
#include "segsum.cuh"

using namespace hb;

namespace {

// Whether the sum of a run updates its rows at once instead of going through memory (write, read, one
// launch).  That saves traffic, but rows are updated where their run ends, a few here and there in a warp,
// while the update kernel takes 32 rows per warp.  For Adagrad it pays where the sums do not fit in L2 (us, at
// once / through memory, ids of Zipf 1.1): 60,000 x 128 77 / 74, 262,144 x 64 of fp16 133 / 119, 120,000 x 128 124 / 114,
// 200,000 x 128 149 / 146, 400,000 x 64 of fp16 154 / 151; 120,000 x 256 158 / 171, 700,000 x 64 231 / 248, 400,000 x 128
// 249 / 263, 1,048,576 x 64 of fp16 284 / 306.
// Adam, with two state rows and two powers per row: 5,000 x 100 47 / 37, 60,000 x 128 84 / 85, 200,000 x 128
// 164 / 144, 700,000 x 128 278 / 268, 1,048,576 x 64 378 / 378: never.
constexpr int64_t kSumsInL2 = 28000000;  // values
bool can_at_once(int64_t dim, const float* grads, const hb_optim_t* opt) {
  if (opt->kind == HB_OPT_ADAM || opt->rows >= ((int64_t)1 << 30)) return false;
  const uintptr_t bits = (uintptr_t)grads | (uintptr_t)opt->emb | (uintptr_t)opt->s0;
  return dim <= seg_tile(dim % 4 == 0 && (bits & 15) == 0);
}
bool at_once(int64_t n, int64_t dim, const float* grads, const hb_optim_t* opt) {
  return n * dim > kSumsInL2 && can_at_once(dim, grads, opt);
}

size_t runs_bytes_of(int64_t n) { return align_up(make_runs_plan(nullptr, n, false).total, 256); }
size_t sums_bytes(int64_t n, int64_t dim) { return align_up((size_t)(n * dim) * sizeof(float), 256); }

}  // namespace

extern "C" {

size_t hb_unique_update_workspace_bytes(int64_t n, int64_t dim, const float* grads, const hb_optim_t* opt) {
  return runs_bytes_of(n) + seg_plan(nullptr, n, dim).total + (at_once(n, dim, grads, opt) ? 0 : sums_bytes(n, dim));
}

int hb_unique_update_f32(const int64_t* ids, const float* grads, const int64_t* cnt_in, int64_t n, const int64_t* n_dev,
                         const int64_t* seg_counts, int64_t seg_cap, int64_t dim, int id_bits, int mean,
                         const hb_optim_t* opt, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31) && dim > 0, "hb_unique_update_f32: bad sizes");
  HB_CHECK_ARG(opt != nullptr && (n == 0 || (ids && grads)), "hb_unique_update_f32: null argument");
  HB_CHECK_ARG(opt->kind == HB_OPT_ADAM || opt->kind == HB_OPT_ADAGRAD, "hb_unique_update_f32: unknown optimiser");
  HB_CHECK_ARG(opt->emb && opt->s0 && (opt->kind != HB_OPT_ADAM || (opt->s1 && opt->step)),
               "hb_unique_update_f32: incomplete optimiser description");
  HB_CHECK_ARG(opt->emb_elem_bytes == 4 || opt->emb_elem_bytes == 2,
               "hb_unique_update_f32: embedding must be fp32 (4) or fp16 (2)");
  HB_CHECK_ARG(opt->rows > 0 && opt->id_stride > 0, "hb_unique_update_f32: bad sizes");
  if (n == 0) return HB_OK;
  // A workspace of a larger batch that is updated at once has no room for the sums: this one is updated at once too.
  const bool can = can_at_once(dim, grads, opt);
  const size_t least = runs_bytes_of(n) + seg_plan(nullptr, n, dim).total;
  const size_t need = least + (can ? 0 : sums_bytes(n, dim));
  if (!workspace || workspace_bytes < need) {
    set_error("hb_unique_update_f32: workspace of %zu bytes needed, %zu given", need, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const bool once = at_once(n, dim, grads, opt) || (can && workspace_bytes < least + sums_bytes(n, dim));
  float* sums = static_cast<float*>(workspace);  // first: on a 256-byte boundary
  char* runs_ws = static_cast<char*>(workspace) + (once ? 0 : sums_bytes(n, dim));
  const size_t runs_bytes = runs_bytes_of(n);
  char* seg_ws = runs_ws + runs_bytes;
  const SegPlan s = seg_plan(seg_ws, n, dim);
  hb_runs_t runs;
  int rc = runs_build(ids, n, n_dev, seg_counts, seg_cap, id_bits, nullptr, 0, nullptr, nullptr, nullptr, nullptr,
                      s.done, s.max_ctas, runs_ws, runs_bytes, &runs, st);
  if (rc != HB_OK) return rc;
  if (!n_dev && !seg_counts) runs.n_dev = nullptr;  // all entries: nothing to wait for
  if (once) {
    SegArgs a = seg_args(&runs, grads, cnt_in, dim, mean, s);
    a.cols = (int)dim;
    const uintptr_t bits = (uintptr_t)grads | (uintptr_t)opt->emb | (uintptr_t)opt->s0;
    return seg_dispatch(a, update_rows<false, false>(&runs, opt), dim % 4 == 0 && (bits & 15) == 0, st);
  }
  rc = segsum_runs(&runs, grads, cnt_in, dim, mean, sums, nullptr, nullptr, seg_ws, s.total, true, true, st);
  if (rc != HB_OK) return rc;
  if (opt->kind == HB_OPT_ADAM)
    return hb_sparse_adam(runs.uniq_ids, sums, nullptr, n, runs.num_runs, dim, opt->id_offset, opt->id_stride, opt->rows,
                          opt->step, opt->s0, opt->s1, opt->emb, opt->emb_elem_bytes, opt->lr, opt->beta1, opt->beta2,
                          opt->eps, stream);
  return hb_sparse_adagrad(runs.uniq_ids, sums, nullptr, n, runs.num_runs, dim, opt->id_offset, opt->id_stride, opt->rows,
                           opt->s0, opt->emb, opt->emb_elem_bytes, opt->lr, opt->eps, stream);
}

}  // extern "C"
