// Segment-sum of gradient rows over runs of equal ids, in one launch: the kernel, and what may
// happen to a finished row (an "epilogue").
//
// Deterministic, no floating-point atomics.  The sorted entries are cut into pieces of R rows; a
// group of G lanes (G * VEC * VPL columns wide) walks its piece in order, reading gradient rows
// through the permutation and adding in registers.
//   * A run that lies inside the piece goes to the epilogue at once.
//   * A run that crosses pieces of one CTA leaves a row per piece in shared memory; after the walk
//     the group where it begins adds them in order.
//   * A run that crosses CTAs leaves one row per CTA in the workspace; the CTA that arrives last
//     (a counter kept at the run's first CTA) adds them: group g takes rows g, g + NG, ..., then
//     the groups' sums are added in order.
// The shapes depend on the sorted order and R only, so two runs on one input give the same bits,
// whichever CTA arrives last.
//
// What bounds it: HBM where there are many rows (2,000,000 x 128: 1.12 GB in 197 us, 5.7 TB/s, 0.89 of
// the measured copy; with the partial rows of every piece in memory and two more launches to add
// them it took 248), latency where there are few (2,000 x 64: 10 us, before 21).
#pragma once

#include "launch.cuh"
#include "maintain.cuh"
#include "optim.cuh"
#include "runs.cuh"

namespace hb {

constexpr int kSegBlockMin = 128;  // threads of the smallest CTA of any epilogue

struct SegArgs {
  const uint8_t* head;        // [n] 1 where a run of equal ids starts in the sorted order
  const int32_t* base8;       // [n / 8] runs that start before entry 8k
  const uint32_t* perm;       // position in the input of each sorted element [n]
  const int64_t* run_start;   // [U + 1] first sorted position of each run; the last: number of valid entries
  const float* grads;         // [n][dim]
  const int64_t* cnt_in;      // nullable [n]
  const int64_t* n_dev;       // nullable device count that caps n
  int64_t n;
  int64_t dim;
  int64_t col0;               // first column of this pass
  int cols;                   // columns of this pass (<= G * VEC * VPL)
  int piece;                  // R: rows per lane group, a power of two
  int mean;                   // divide by the count
  int early;                  // the launch before is one of this call's: blocks may take their places under it (HB_LAUNCH_NEXT)
  // per CTA: what its part of a run that began earlier / of its last run adds up to
  float* head_part;           // [CTAs][cols]
  float* tail_part;           // [CTAs][cols]
  unsigned long long* head_cnt;  // [CTAs] (weights given)
  unsigned long long* tail_cnt;  // [CTAs]
  unsigned* done;             // [CTAs] zero before and after: arrivals of the run that begins in the CTA
};

// hb_segsum_runs_f32; zeroed: the arrival counters are at zero already; early: SegArgs
int segsum_runs(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim, int mean, float* sums,
                int64_t* counts, const hb_class_split_t* split, void* workspace, size_t workspace_bytes, bool zeroed,
                bool early, cudaStream_t st);

// ---- epilogues ---------------------------------------------------------------------------------
// The sums and counts as they are, or the buffers of the id's class.
struct StoreRows {
  static constexpr bool kWeights = true;
  static constexpr bool kStep = false;
  float* sums;                // [U][dim] (null when the rows go to class buffers)
  const int8_t* dclass;       // [U], null = no split
  const int32_t* dpos;        // [U]
  float* class_rows[3];
  int64_t* counts;            // [U], nullable
  int64_t* class_counts[3];   // per class, nullable
};

// The row is a gradient: update the optimiser state and the table row of its id.  STEP (the
// one-trainer step): HOT rows are updated, COLD rows are added to their staging slots.  Fewer than
// 2^30 rows and slots.
template <bool ADAM, bool STEP>
struct UpdateRows {
  static constexpr bool kAdam = ADAM;
  static constexpr bool kStep = STEP;
  static constexpr bool kWeights = !STEP;  // rows with weights come from several senders
  const int64_t* uniq;        // [U] ids
  RowMap map;
  int half;                   // fp16 rows
  float* step;
  float* s0;
  float* s1;
  void* emb;
  AdamParams p;
  // STEP only
  float* sums;                // [U][dim], where updates come behind the sums (SegWalk)
  const int8_t* dclass;       // [U]
  float* staged;              // [slots][dim]
  const int64_t* slots;       // [U] staging slot of a cold run, -1 = none
  // blocks that age the LRU counters by the lookup that found the slots: the first of the sums' launch, the last of the
  // second pass's
  int touch_blocks;
  RunsView touched;
  TouchMarks marks;
  int32_t* lru;
};

template <bool ADAM, bool STEP>
UpdateRows<ADAM, STEP> update_rows(const hb_runs_t* runs, const hb_optim_t* opt) {
  UpdateRows<ADAM, STEP> epi;
  epi.uniq = runs->uniq_ids;
  epi.map = RowMap{opt->id_offset, opt->id_stride, opt->rows};
  epi.half = opt->emb_elem_bytes == 2;
  epi.step = opt->step;
  epi.s0 = opt->s0;
  epi.s1 = opt->s1;
  epi.emb = opt->emb;
  epi.p = AdamParams{(float)opt->lr, (float)opt->beta1, (float)opt->beta2, (float)opt->eps,
                     (float)(1.0 - opt->beta1), (float)(1.0 - opt->beta2)};
  epi.sums = nullptr;
  epi.dclass = nullptr;
  epi.staged = nullptr;
  epi.slots = nullptr;
  epi.touch_blocks = 0;
  return epi;
}

#ifdef __CUDACC__

template <int VEC> struct VecF;
template <> struct VecF<4> { using T = float4; };
template <> struct VecF<1> { using T = float; };

__device__ __forceinline__ void vadd(float4& a, const float4& b) {
  a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
}
__device__ __forceinline__ void vadd(float& a, const float& b) { a += b; }
__device__ __forceinline__ void vzero(float4& a) { a = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void vzero(float& a) { a = 0.f; }
// a / d for a whole number d with r = 1 / d given: one correction of the product by its remainder, which is
// exact as d is whole (Markstein: the quotient is then correctly rounded; a subnormal one that lies halfway
// between two floats goes to either), instead of a division per value.  The remainder of an infinite sum is NaN, of
// which the minimum makes a number that leaves the infinity as it is.  (60,000 rows for Adam, sums and update: 84.2
// us without, 84.7 so, with a select 2 % more, with a branch to a division 5 %: registers.)
__device__ __forceinline__ void vdiv(float& a, float d, float r) {
  const float q = a * r;
  a = fmaf(fminf(fmaf(-q, d, a), 3.402823466e38f), r, q);
}
__device__ __forceinline__ void vdiv(float4& a, float d, float r) {
  vdiv(a.x, d, r);
  vdiv(a.y, d, r);
  vdiv(a.z, d, r);
  vdiv(a.w, d, r);
}
__device__ __forceinline__ float& lane_of(float4& a, int j) { return reinterpret_cast<float*>(&a)[j]; }
__device__ __forceinline__ float& lane_of(float& a, int) { return a; }

__device__ __forceinline__ void l2_prefetch_row(const void* row, int bytes) {
  const char* p = static_cast<const char*>(row);
  for (int at = 0; at < bytes; at += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + at));
}

// What the kernel asks of an epilogue, for rows spread over the G lanes of a group (acc[v] is vector
// sub + v * G):
//   Lane        what a lane finds out about the run that ends at its entry
//   Row         what has to be in registers to finish a run; fetched with the gradient rows, for
//               every run that ends among the kFly entries in flight
//   finish      the complete row
template <class Epi, int VEC, int G, int VPL> struct EpiOps;

template <int VEC, int G, int VPL>
struct EpiOps<StoreRows, VEC, G, VPL> {
  using V = typename VecF<VEC>::T;
  static constexpr int kFly = (8 / VPL) < G ? (8 / VPL) : G;
  static constexpr int kBlock = 256;
  static constexpr int kMinBlocks = 4;  // (rows of 128 columns: 64 registers and 30 bytes of spills; with weights 68)
  static constexpr int kPieceMax = 32;
  static constexpr bool kPrefetch = false;
  struct Lane {};
  struct Row {};
  static __device__ __forceinline__ Lane lane(const StoreRows&, int) { return Lane(); }
  static __device__ __forceinline__ void prefetch(const StoreRows&, const SegArgs&, const Lane&) {}
  static __device__ __forceinline__ void fetch(const StoreRows&, const SegArgs&, const Lane&, int, bool, int, int, Row&) {}
  static __device__ __forceinline__ Row fetch_alone(const StoreRows&, const SegArgs&, int, int, int) { return Row(); }
  static __device__ __forceinline__ void finish(const StoreRows& o, const SegArgs& a, int64_t u, V (&acc)[VPL],
                                                Row&, int sub, int vpr, long long count) {
    float* base = o.sums;
    int64_t row = u;
    int64_t* counts = o.counts;
    if (o.dclass) {
      const int c = o.dclass[u];
      base = c == 0 ? o.class_rows[0] : (c == 1 ? o.class_rows[1] : (c == 2 ? o.class_rows[2] : nullptr));
      counts = c == 0 ? o.class_counts[0] : (c == 1 ? o.class_counts[1] : (c == 2 ? o.class_counts[2] : nullptr));
      row = o.dpos[u];
    }
    if (base) {
      V* dst = reinterpret_cast<V*>(base + row * a.dim + a.col0);
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        const int k = sub + v * G;
        if (k < vpr) dst[k] = acc[v];
      }
    }
    if (counts && sub == 0 && a.col0 == 0) counts[row] = count;
  }
};

template <int VEC>
__device__ __forceinline__ typename VecF<VEC>::T load_emb(const void* p, int64_t at, bool half);
template <>
__device__ __forceinline__ float4 load_emb<4>(const void* p, int64_t at, bool half) {
  return half ? EmbIO<__half>::load4(reinterpret_cast<const __half*>(p) + at)
              : EmbIO<float>::load4(reinterpret_cast<const float*>(p) + at);
}
template <>
__device__ __forceinline__ float load_emb<1>(const void* p, int64_t at, bool half) {
  return half ? EmbIO<__half>::load(reinterpret_cast<const __half*>(p) + at)
              : EmbIO<float>::load(reinterpret_cast<const float*>(p) + at);
}
__device__ __forceinline__ void store_emb(void* p, int64_t at, bool half, const float4& v) {
  if (half) EmbIO<__half>::store4(reinterpret_cast<__half*>(p) + at, v);
  else EmbIO<float>::store4(reinterpret_cast<float*>(p) + at, v);
}
__device__ __forceinline__ void store_emb(void* p, int64_t at, bool half, float v) {
  if (half) EmbIO<__half>::store(reinterpret_cast<__half*>(p) + at, v);
  else EmbIO<float>::store(reinterpret_cast<float*>(p) + at, v);
}

// The rows to update are scattered over memory and most runs are short: fetched one after the
// other, each when its sum is complete, they cost a memory latency per run (1,048,576 gradients of 64
// columns for fp16 rows: 826 us).  So every lane looks up the row of the run that ends at its own
// entry, all lanes prefetch their gradient, state and table rows into L2, and the walk over the
// entries finds them there with few registers per entry in flight: the arithmetic (two or three IEEE
// divisions and a square root per value) needs the warps.
template <bool ADAM, bool STEP, int VEC, int G, int VPL>
struct EpiOps<UpdateRows<ADAM, STEP>, VEC, G, VPL> {
  using V = typename VecF<VEC>::T;
  using Epi = UpdateRows<ADAM, STEP>;
  static constexpr int kStaged = 1 << 30;  // added to a row number: a staging slot
  static constexpr int kFly = VPL == 1 ? 2 : 1;
  // (a step's sums have the bits of StoreRows: a captured step and an eager one may differ in which they use)
  static constexpr int kBlock = STEP ? 256 : 128;
  static constexpr int kMinBlocks = (VPL > 2 ? 512 : 768) / kBlock;
  static constexpr int kPieceMax = STEP ? 32 : 16;
  static constexpr bool kPrefetch = true;
  // per-row scalars divide where the stand-alone kernels do (columns one by one), else their reciprocals multiply
  static constexpr bool kDivide = VEC == 1;
  struct Lane {
    int row = -1;   // table row, or kStaged + staging slot
    float t = 0.0f, ra = 1.0f, rb = 1.0f;  // the bias corrections or their reciprocals
  };
  struct Row {
    int row;
    float t, ra, rb;
    V e[VPL], s0[VPL], s1[ADAM ? VPL : 1];
  };
  static __device__ __forceinline__ bool is_staged(int row) { return STEP && row >= kStaged; }
  static __device__ __forceinline__ int row_of(const Epi& o, int64_t run) {
    // (all on their way before one of them decides)
    const int64_t id = o.uniq[run], slot = STEP ? o.slots[run] : -1;
    const int c = STEP ? o.dclass[run] : 1;
    if (STEP && c == 2) return slot >= 0 ? kStaged + (int)slot : -1;
    return c == 1 ? (int)o.map(id) : -1;
  }
  static __device__ __forceinline__ Lane lane(const Epi& o, int64_t run) {
    Lane l;
    l.row = row_of(o, run);
    if (ADAM && l.row >= 0 && !is_staged(l.row)) {
      // state_step = state_step + 1 (per row), sparse_optim.py:624-626
      l.t = o.step[l.row] + 1.0f;
      l.ra = 1.0f - powf(o.p.beta1, l.t);
      l.rb = 1.0f - powf(o.p.beta2, l.t);
      if (!kDivide) {
        l.ra = 1.0f / l.ra;
        l.rb = 1.0f / l.rb;
      }
    }
    return l;
  }
  static __device__ __forceinline__ void prefetch(const Epi& o, const SegArgs& a, const Lane& l) { prefetch(o, a, l.row); }
  static __device__ __forceinline__ void prefetch(const Epi& o, const SegArgs& a, int row) {
    if (row < 0) return;
    if (is_staged(row)) {
      l2_prefetch_row(o.staged + (int64_t)(row - kStaged) * a.dim, (int)a.dim * 4);
      return;
    }
    const int64_t at = (int64_t)row * a.dim;
    l2_prefetch_row(o.s0 + at, (int)a.dim * 4);
    if (ADAM) l2_prefetch_row(o.s1 + at, (int)a.dim * 4);
    l2_prefetch_row(reinterpret_cast<const char*>(o.emb) + at * (o.half ? 2 : 4), (int)a.dim * (o.half ? 2 : 4));
  }
  static __device__ __forceinline__ void load(const Epi& o, const SegArgs& a, int sub, int vpr, Row& r) {
    if (r.row < 0) return;
    const bool st = is_staged(r.row);
    const int64_t at = (int64_t)(st ? r.row - kStaged : r.row) * a.dim + sub * VEC;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (sub + v * G >= vpr) continue;
      const int64_t k = at + v * G * VEC;
      if (st) {
        r.e[v] = *reinterpret_cast<const V*>(o.staged + k);
      } else {
        r.s0[v] = *reinterpret_cast<const V*>(o.s0 + k);
        if (ADAM) r.s1[v] = *reinterpret_cast<const V*>(o.s1 + k);
        r.e[v] = load_emb<VEC>(o.emb, k, o.half);
      }
    }
  }
  // by all lanes of the warp: the run that ends at the entry of lane `src` of each W lanes
  template <int W = G>
  static __device__ __forceinline__ void fetch(const Epi& o, const SegArgs& a, const Lane& l, int src, bool ends, int sub,
                                               int vpr, Row& r) {
    r.row = __shfl_sync(0xffffffffu, l.row, src, W);
    if (ADAM) {
      r.t = __shfl_sync(0xffffffffu, l.t, src, W);
      r.ra = __shfl_sync(0xffffffffu, l.ra, src, W);
      r.rb = __shfl_sync(0xffffffffu, l.rb, src, W);
    }
    if (ends) load(o, a, sub, vpr, r);
  }
  static __device__ __forceinline__ Row fetch_alone(const Epi& o, const SegArgs& a, int run, int sub, int vpr) {
    const Lane l = lane(o, run);  // the same in every lane of the group
    Row r;
    r.row = l.row;
    r.t = l.t;
    r.ra = l.ra;
    r.rb = l.rb;
    load(o, a, sub, vpr, r);
    return r;
  }
  static __device__ __forceinline__ void finish(const Epi& o, const SegArgs& a, int64_t, V (&acc)[VPL], Row& r, int sub,
                                                int vpr, long long count) {
    if (r.row < 0) return;
    const bool st = is_staged(r.row);
    const int64_t at = (int64_t)(st ? r.row - kStaged : r.row) * a.dim + sub * VEC;
    if (st) {
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        if (sub + v * G >= vpr) continue;
        vadd(r.e[v], acc[v]);
        *reinterpret_cast<V*>(o.staged + at + v * G * VEC) = r.e[v];
      }
      return;
    }
    // one trainer: unique_grads of its own rows divides by 1 + their count
    const float c = STEP ? (float)(count + 1) : 1.0f, rc = kDivide ? 1.0f : 1.0f / c;
    if (ADAM && sub == 0) o.step[r.row] = r.t;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      if (sub + v * G >= vpr) continue;
#pragma unroll
      for (int j = 0; j < VEC; ++j) {
        const float sum = lane_of(acc[v], j);
        const float g = !STEP ? sum : kDivide ? sum / c : sum * rc;
        if constexpr (ADAM && kDivide)
          lane_of(r.e[v], j) -= adam_elem(g, lane_of(r.s0[v], j), lane_of(r.s1[v], j), r.ra, r.rb, o.p);
        else if constexpr (ADAM) adam_value(g, lane_of(r.s0[v], j), lane_of(r.s1[v], j), lane_of(r.e[v], j), r.ra, r.rb, o.p);
        else adagrad_value(g, lane_of(r.s0[v], j), lane_of(r.e[v], j), o.p);
      }
      const int64_t k = at + v * G * VEC;
      *reinterpret_cast<V*>(o.s0 + k) = r.s0[v];
      if constexpr (ADAM) *reinterpret_cast<V*>(o.s1 + k) = r.s1[v];
      store_emb(o.emb, k, o.half, r.e[v]);
    }
  }
};

// Runs first .. first + runs, whose sums are in sums[run], by `nwarps` warps side by side in chunks of eight: a lane
// each for what is worked out once per id, then G lanes per row.
template <bool ADAM, int VEC, int G, int VPL>
__device__ __forceinline__ void apply_runs(const UpdateRows<ADAM, true>& o, const SegArgs& a, const float* sums, int64_t first,
                                           int64_t runs, int64_t warp, int64_t nwarps) {
  using V = typename VecF<VEC>::T;
  using Ops = EpiOps<UpdateRows<ADAM, true>, VEC, G, VPL>;
  constexpr int RPP = 32 / G, kChunk = 8;
  const int lane = threadIdx.x & 31;
  const int sub = lane & (G - 1), which = lane / G;
  const int vpr = a.cols / VEC;
  auto run_of = [&](int64_t chunk, int q) { return ((chunk + q / kChunk) * nwarps + warp) * kChunk + q % kChunk; };
  for (int64_t chunk = 0; run_of(chunk, 0) < runs; chunk += 32 / kChunk) {
    const int64_t u = run_of(chunk, lane);
    typename Ops::Lane mine;
    int count = 0;
    if (u < runs) {
      count = (int)(a.run_start[first + u + 1] - a.run_start[first + u]);
      mine = Ops::lane(o, first + u);
    }
    const unsigned some = __ballot_sync(0xffffffffu, mine.row >= 0);
    for (int t0 = 0; t0 < 32 && (some >> t0) != 0u; t0 += RPP) {
      const int q = t0 + which;
      V acc[VPL];
      typename Ops::Row with;
      const int cnt = __shfl_sync(0xffffffffu, count, q);
      Ops::template fetch<32>(o, a, mine, q, true, sub, vpr, with);
      if (with.row < 0) continue;
      const V* src = reinterpret_cast<const V*>(sums + (first + run_of(chunk, q)) * a.dim);
#pragma unroll
      for (int k = 0; k < VPL; ++k)
        if (sub + k * G < vpr) acc[k] = __ldcg(src + sub + k * G);
      Ops::finish(o, a, 0, acc, with, sub, vpr, cnt);
    }
  }
}

// What the walk over the entries does with complete rows: the epilogue at once, or, for Adam in a step, they are stored
// in the shape of StoreRows (a captured step and an eager one may differ in which they use), and the CTA updates their rows
// when it has them all.  An update where a run ends holds up the lane groups whose runs go on, and where runs are of
// very different lengths most warps wait for a few; behind the sums every warp has its share (us a step without flushes,
// in the walk / behind it: 10,000 x 64 63.1 / 58.9, 50,000 x 32 83.1 / 76.4, 65,536 x 128 111.0 / 107.5;
// Adagrad, with half the values and half the arithmetic, 65,536 x 128 102.9 / 103.7.  With all lanes of a warp on one row and 32 warps an SM: 50,000 x 128 of next to no
// duplicates 106.4 / 108.4, now 104.5).
template <class Epi, int VEC, int G, int VPL> struct SegWalk {
  using Ops = EpiOps<Epi, VEC, G, VPL>;
  static constexpr bool kBehind = false;
  static constexpr int kMinBlocks = Ops::kMinBlocks;
  static __device__ __forceinline__ const Epi& out(const Epi& epi) { return epi; }
};
template <int VEC, int G, int VPL> struct SegWalk<UpdateRows<true, true>, VEC, G, VPL> {
  using Ops = EpiOps<StoreRows, VEC, G, VPL>;
  static constexpr int kMinBlocks = VPL > 2 ? 2 : 3;
  static constexpr bool kBehind = true;
  static __device__ __forceinline__ StoreRows out(const UpdateRows<true, true>& epi) {
    StoreRows o = {};
    o.sums = epi.sums;
    return o;
  }
};

// ---- the kernel ----------------------------------------------------------------------------------
constexpr unsigned char kSegHead = 1;    // the piece begins inside a run: a row in s_head
constexpr unsigned char kSegWhole = 2;   // ... which goes on behind the piece
constexpr unsigned char kSegTail = 4;    // the piece's last run begins in it and goes on behind it

template <int VEC, int G, int VPL, bool HAS_CNT, class Epi>
__global__ void __launch_bounds__(SegWalk<Epi, VEC, G, VPL>::Ops::kBlock, SegWalk<Epi, VEC, G, VPL>::kMinBlocks)
segsum_kernel(SegArgs a, Epi epi) {
  begin_after_previous();
  using V = typename VecF<VEC>::T;
  using Walk = SegWalk<Epi, VEC, G, VPL>;
  using Ops = typename Walk::Ops;
  const auto& out = Walk::out(epi);
  constexpr int NG = Ops::kBlock / G;
  constexpr int U = Ops::kFly;  // rows whose loads are in flight together
  extern __shared__ __align__(16) float s_rows[];   // [NG][cols] pieces' parts of a run that began earlier
  __shared__ unsigned char s_flag[NG];
  __shared__ unsigned long long s_cnt[HAS_CNT ? NG : 1];
  __shared__ int s_fin_run[2], s_fin_first[2], s_fin_parts[2];
  __shared__ int s_nfin;
  const int lane = threadIdx.x & 31;
  const int sub = lane & (G - 1);
  const int grp = threadIdx.x / G;
  const unsigned shift = (lane / G) * G;
  const unsigned gbits = G == 32 ? 0xffffffffu : ((1u << G) - 1u);
  const unsigned gmask = gbits << shift;
  int n_eff = (int)a.n;
  if (a.n_dev) {
    const int64_t d = *a.n_dev;
    n_eff = d < a.n ? (d > 0 ? (int)d : 0) : (int)a.n;
  }
  const int R = a.piece;
  const int span = NG * R;
  int block = blockIdx.x;
  if constexpr (Epi::kStep) {
    if (block < epi.touch_blocks) {
      touch_runs(epi.touched, epi.marks, epi.lru, block, epi.touch_blocks);
      return;
    }
    block -= epi.touch_blocks;
  }
  const int64_t b0 = (int64_t)block * span;
  if (b0 >= n_eff) return;
  // what the sort found (in a step the lookup of the cold ids comes between)
  auto found = [](const auto* p) {
    if constexpr (Epi::kStep) return load_settled(p);
    else return *p;
  };
  if (threadIdx.x == 0) s_nfin = 0;
  const int64_t at = b0 + (int64_t)grp * R;
  const bool live = at < n_eff;
  const int j0 = live ? (int)at : n_eff;
  const int len = n_eff - j0 < R ? n_eff - j0 : R;  // (j0 + R may not be a number: entries are counted from j0)
  const int vpr = a.cols / VEC;  // vectors per row in this pass

  // The runs that begin and end in this CTA, which it updates once they are summed up: their state and table rows are on
  // their way to L2 meanwhile.
  int run0 = 0, runs = 0;
  if constexpr (Walk::kBehind) {
    auto begun = [&](int j) {  // runs that begin at entry j or before it
      const unsigned long long f = *reinterpret_cast<const unsigned long long*>(a.head + (j & ~7));
      return found(a.base8 + (j >> 3)) + __popcll(f & (~0ull >> (8 * (7 - (j & 7)))));
    };
    const int e = n_eff - (int)b0 < span ? n_eff : (int)b0 + span;  // (b0 + span may not be a number)
    run0 = begun((int)b0) - (found(a.head + b0) != 0);
    runs = begun(e - 1) - 1 + (e == n_eff || found(a.head + e) != 0) - run0;
    using Rows = EpiOps<Epi, VEC, G, VPL>;
    for (int r = threadIdx.x; r < runs; r += Ops::kBlock) Rows::prefetch(epi, a, Rows::row_of(epi, run0 + r));
  }

  int u = -1;              // the open run; before the first head of a piece that begins with one: the run before
  bool first_partial = false;
  if (live) {
    // head flags of the 8 entries around j0 (pieces of a narrow row may begin inside them)
    const unsigned long long f = *reinterpret_cast<const unsigned long long*>(a.head + (j0 & ~7));
    first_partial = ((f >> (8 * (j0 & 7))) & 1ull) == 0ull;
    u = found(a.base8 + (j0 >> 3)) - 1 + __popcll(f & ((1ull << (8 * (j0 & 7))) - 1ull));
  }
  const int u_first = u;
  bool open = first_partial;  // a run is open
  V acc[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) vzero(acc[v]);
  unsigned long long cacc = 0;
  unsigned char flag = 0;

  // a run is complete: its row (and count) to the epilogue
  auto complete = [&](int run, V (&row)[VPL], typename Ops::Row& with, unsigned long long weight) {
    long long count = (long long)weight;
    if (a.mean) {
      // unique_grads starts its counts from ones when cnt is given (sparse_optim.py:145-148)
      if (HAS_CNT) count += 1;
      const float d = (float)count, r = 1.0f / d;
#pragma unroll
      for (int v = 0; v < VPL; ++v) vdiv(row[v], d, r);
    }
    Ops::finish(out, a, run, row, with, sub, vpr, count);
  };
  auto put = [&](float* dst, const V (&row)[VPL]) {
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int k = sub + v * G;
      if (k < vpr) reinterpret_cast<V*>(dst)[k] = row[v];
    }
  };
  auto add = [&](V (&row)[VPL], const float* src) {
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      const int k = sub + v * G;
      if (k < vpr) vadd(row[v], reinterpret_cast<const V*>(src)[k]);
    }
  };

  const int eg = R < G ? R : G;                 // entries per step
  const int steps = (R + eg - 1) / eg;
  uint32_t p_next = 0;
  bool head_next = false, end_next = false;
  auto look = [&](int j) {  // entry j of the sorted order
    p_next = found(a.perm + j);
    head_next = found(a.head + j) != 0;
    end_next = j + 1 >= n_eff || found(a.head + j + 1) != 0;
  };
  if (sub < eg && sub < len) look(j0 + sub);
  for (int s = 0; s < steps; ++s) {
    const int at = s * eg + sub;
    const bool valid = sub < eg && at < len;
    const uint32_t p = p_next;
    const unsigned heads = (__ballot_sync(0xffffffffu, valid && head_next) >> shift) & gbits;
    const unsigned ends = (__ballot_sync(0xffffffffu, valid && end_next) >> shift) & gbits;
    const unsigned valids = (__ballot_sync(0xffffffffu, valid) >> shift) & gbits;
    typename Ops::Lane mine;
    // (a run that began before the piece is not finished by this group)
    if ((ends >> sub) & 1u) {
      const int begun = __popc(heads & ((2u << sub) - 1u));
      if (begun || !first_partial) mine = Ops::lane(out, u + begun);
    }
    int cv = 1;
    if (HAS_CNT && valid) cv = (int)a.cnt_in[p];
    if (Ops::kPrefetch && valid) {
      l2_prefetch_row(a.grads + (int64_t)p * a.dim + a.col0, a.cols * 4);
      Ops::prefetch(out, a, mine);
    }
    if (s + 1 < steps && sub < eg && at + eg < len) look(j0 + at + eg);
#pragma unroll 1
    for (int t0 = 0; t0 < eg; t0 += U) {
      V val[U][VPL];
      typename Ops::Row with[U];
      int cvs[U];
#pragma unroll
      for (int x = 0; x < U; ++x) {
        const uint32_t px = __shfl_sync(0xffffffffu, p, t0 + x, G);
        cvs[x] = HAS_CNT ? __shfl_sync(0xffffffffu, cv, t0 + x, G) : 1;
        if ((valids >> (t0 + x)) & 1u) {
          const V* src = reinterpret_cast<const V*>(a.grads + (int64_t)px * a.dim + a.col0);
#pragma unroll
          for (int v = 0; v < VPL; ++v) {
            const int k = sub + v * G;
            if (k < vpr) val[x][v] = load_settled(src + k);
          }
        }
        Ops::fetch(out, a, mine, t0 + x, (ends >> (t0 + x)) & 1u, sub, vpr, with[x]);
      }
#pragma unroll
      for (int x = 0; x < U; ++x) {
        if (!((valids >> (t0 + x)) & 1u)) continue;
        if ((heads >> (t0 + x)) & 1u) {
          ++u;
          open = true;
#pragma unroll
          for (int v = 0; v < VPL; ++v) vzero(acc[v]);
          cacc = 0;
        }
#pragma unroll
        for (int v = 0; v < VPL; ++v) {
          const int k = sub + v * G;
          if (k < vpr) vadd(acc[v], val[x][v]);
        }
        cacc += (unsigned long long)(unsigned)cvs[x];
        if ((ends >> (t0 + x)) & 1u) {
          if (first_partial) {
            put(s_rows + grp * a.cols, acc);
            if (HAS_CNT && sub == 0) s_cnt[grp] = cacc;
            flag |= kSegHead;
            first_partial = false;
          } else {
            complete(u, acc, with[x], cacc);
          }
          open = false;
        }
      }
    }
  }
  if (open) {  // the last run goes on behind the piece
    if (first_partial) {
      put(s_rows + grp * a.cols, acc);
      if (HAS_CNT && sub == 0) s_cnt[grp] = cacc;
      flag |= kSegHead | kSegWhole;
    } else {
      flag |= kSegTail;
    }
  }
  if (sub == 0) s_flag[grp] = flag;
  __syncthreads();

  // this CTA's part of a run that crosses CTAs is in the workspace: has every other part arrived?
  auto arrive = [&](int run) {
    const int first = (int)(found(a.run_start + run) / span);
    const int last = (int)((found(a.run_start + run + 1) - 1) / span);
    __threadfence();
    __syncwarp(gmask);
    if (sub == 0) {
      const int parts = last - first + 1;
      if ((int)atomicAdd(a.done + first, 1u) == parts - 1) {
        const int at = atomicAdd(&s_nfin, 1);  // at most two per CTA, in any order: they are different runs
        s_fin_run[at] = run;
        s_fin_first[at] = first;
        s_fin_parts[at] = parts;
      }
    }
  };
  if (grp == 0 && (flag & kSegHead)) {
    V row[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) vzero(row[v]);
    unsigned long long w = 0;
    for (int g = 0; g < NG; ++g) {
      add(row, s_rows + g * a.cols);
      if (HAS_CNT) w += s_cnt[g];
      if (!(s_flag[g] & kSegWhole)) break;
    }
    put(a.head_part + (int64_t)block * a.cols, row);
    if (HAS_CNT && sub == 0) a.head_cnt[block] = w;
    arrive(u_first);
  }
  if (flag & kSegTail) {
    bool ended = false;
    for (int g = grp + 1; g < NG; ++g) {
      add(acc, s_rows + g * a.cols);
      if (HAS_CNT) cacc += s_cnt[g];
      if (!(s_flag[g] & kSegWhole)) { ended = true; break; }
    }
    if (ended) {
      typename Ops::Row with = Ops::fetch_alone(out, a, u, sub, vpr);
      complete(u, acc, with, HAS_CNT ? cacc : (unsigned long long)(found(a.run_start + u + 1) - found(a.run_start + u)));
    } else {
      put(a.tail_part + (int64_t)block * a.cols, acc);
      if (HAS_CNT && sub == 0) a.tail_cnt[block] = cacc;
      arrive(u);
    }
  }
  __syncthreads();
  const int nfin = s_nfin;
  for (int f = 0; f < nfin; ++f) {
    __threadfence();
    const int run = s_fin_run[f], first = s_fin_first[f], parts = s_fin_parts[f];
    V row[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) vzero(row[v]);
    unsigned long long w = 0;
    constexpr int kFly = VPL == 1 ? 8 : (VPL == 2 ? 4 : 2);
    for (int i0 = grp; i0 < parts; i0 += NG * kFly) {
      V x[kFly][VPL];
#pragma unroll
      for (int q = 0; q < kFly; ++q) {
        const int i = i0 + q * NG;
        if (i >= parts) continue;
        const float* src = (i == 0 ? a.tail_part : a.head_part) + (int64_t)(first + i) * a.cols;
#pragma unroll
        for (int v = 0; v < VPL; ++v)
          if (sub + v * G < vpr) x[q][v] = __ldcg(reinterpret_cast<const V*>(src) + sub + v * G);
        if (HAS_CNT) w += __ldcg((i == 0 ? a.tail_cnt : a.head_cnt) + first + i);
      }
#pragma unroll
      for (int q = 0; q < kFly; ++q) {
        if (i0 + q * NG >= parts) continue;
#pragma unroll
        for (int v = 0; v < VPL; ++v)
          if (sub + v * G < vpr) vadd(row[v], x[q][v]);
      }
    }
    put(s_rows + grp * a.cols, row);
    if (HAS_CNT && sub == 0) s_cnt[grp] = w;
    __syncthreads();
    if (grp == 0) {
      for (int g = 1; g < NG && g < parts; ++g) {
        add(row, s_rows + g * a.cols);
        if (HAS_CNT) w += s_cnt[g];
      }
      typename Ops::Row with = Ops::fetch_alone(out, a, run, sub, vpr);
      complete(run, row, with, HAS_CNT ? w : (unsigned long long)(found(a.run_start + run + 1) - found(a.run_start + run)));
      if (sub == 0) a.done[first] = 0u;
    }
    __syncthreads();
  }
  if constexpr (Walk::kBehind) {
    constexpr int W = Ops::kBlock / 32;
    const int warp = threadIdx.x >> 5;
    for (int f = 0; f < nfin; ++f)  // runs that crossed CTAs: a warp each, of those that may have fewer of the others
      if (warp == W - 1 - f) apply_runs<Epi::kAdam, VEC, G, VPL>(epi, a, epi.sums, s_fin_run[f], 1, 0, 1);
    apply_runs<Epi::kAdam, VEC, G, VPL>(epi, a, epi.sums, run0, runs, warp, W);
  }
}

// ---- host side ------------------------------------------------------------------------------------
// Rows per lane group: short pieces while the GPU has room for more groups (a piece is a chain of
// loads), up to kPieceMax once every SM has its 32 warps.  Measured on 2,000,000 x 128 (us, sums): 8: 224,
// 16: 198, 32: 197, 64: 205; on 1,048,576 x 64 with the update fused: 235, 222, 239, 279 (16 in CTAs of 128
// threads instead of 32 in CTAs of 256: the whole call 314 -> 291, with 3 to 5 % on other widths; CTAs of 128
// cost the plain sums of 2,000 x 64 2 us).  The shortest, 4: with 8 a step of 2,000 x 64 takes 66 us instead of
// 62, of 20,000 x 128 91 instead of 87, sums of 30,000 x 128 14.4 instead of 11.2.
constexpr int kPieceMin = 4;
static inline int seg_piece(int64_t n, int lanes_per_row, int most) {
  int r = kPieceMin;
  while (r < most && ceil_div(n, r) * lanes_per_row / 32 > (int64_t)sm_count() * 32) r *= 2;
  return r;
}

struct SegPlan {
  float *head_part, *tail_part;
  unsigned long long *head_cnt, *tail_cnt;
  unsigned* done;
  int64_t max_ctas;
  size_t total;
};

static inline SegPlan seg_plan(void* ws, int64_t n, int64_t dim) {
  SegPlan s;
  Carver cv(ws ? ws : (void*)256);  // a null workspace still yields the sizes
  const int64_t m = n > 0 ? n : 1;
  // CTAs of 4 groups (32 lanes per row) or more; pieces of 8 rows or longer, shorter ones only while the
  // groups do not fill the GPU (a bound that does not fall with n: a workspace serves smaller batches)
  s.max_ctas = ceil_div(m, 8 * (kSegBlockMin / 32));
  const int64_t few = ceil_div(m, kPieceMin * (kSegBlockMin / 32)), filled = (int64_t)sm_count() * 64;
  if (s.max_ctas < few) s.max_ctas = s.max_ctas > filled ? s.max_ctas : (few < filled ? few : filled);
  s.max_ctas += 1;
  const size_t cols = (size_t)(dim < 512 ? dim : 512);
  s.head_part = cv.take<float>((size_t)s.max_ctas * cols);
  s.tail_part = cv.take<float>((size_t)s.max_ctas * cols);
  s.head_cnt = cv.take<unsigned long long>(s.max_ctas);
  s.tail_cnt = cv.take<unsigned long long>(s.max_ctas);
  s.done = cv.take<unsigned>(s.max_ctas);
  s.total = cv.used() + 256;
  return s;
}

template <int VEC, int G, int VPL, class Epi>
int seg_launch(SegArgs a, const Epi& epi, cudaStream_t st) {
  using Ops = typename SegWalk<Epi, VEC, G, VPL>::Ops;
  a.piece = seg_piece(a.n, G, Ops::kPieceMax);
  const int ng = Ops::kBlock / G;
  int grid = (int)ceil_div(a.n, (int64_t)ng * a.piece);
  if constexpr (Epi::kStep) grid += epi.touch_blocks;
  const size_t smem = (size_t)ng * a.cols * sizeof(float);
  // Behind a sort of the whole GPU blocks that take their places early find the SMs set up for its 200 KB of shared
  // memory, and next to no L1 for their rows (524,288 x 128: 64 -> 78 us).
  const bool early = a.early && a.n <= kSortClusterEntries;
#define HB_SEG(CNT)                                                                                     \
  do {                                                                                                  \
    if (early) HB_LAUNCH_NEXT((segsum_kernel<VEC, G, VPL, CNT, Epi>), grid, Ops::kBlock, smem, st, a, epi); \
    else HB_LAUNCH((segsum_kernel<VEC, G, VPL, CNT, Epi>), grid, Ops::kBlock, smem, st, a, epi);        \
  } while (0)
  if constexpr (Epi::kWeights) {
    if (a.cnt_in) {
      HB_SEG(true);
      return HB_OK;
    }
  }
  HB_SEG(false);
#undef HB_SEG
  return HB_OK;
}

template <class Epi>
int seg_dispatch(const SegArgs& a, const Epi& epi, bool vec4, cudaStream_t st) {
  // Two vectors per lane and half the lanes per row: what is done per entry and not per value
  // (addresses, shuffles, masks) is as many instructions as the arithmetic of one vector.
  if (vec4) {
    const int vpr = a.cols / 4;
    if (vpr > 64) return seg_launch<4, 32, 4>(a, epi, st);
    if (vpr > 32) return seg_launch<4, 32, 2>(a, epi, st);
    if (vpr > 16) return seg_launch<4, 16, 2>(a, epi, st);
    if (vpr > 8) return seg_launch<4, 8, 2>(a, epi, st);
    return seg_launch<4, 4, 2>(a, epi, st);
  }
  const int vpr = a.cols;
  if (vpr > 64) return seg_launch<1, 32, 4>(a, epi, st);
  if (vpr > 32) return seg_launch<1, 32, 2>(a, epi, st);
  if (vpr > 16) return seg_launch<1, 32, 1>(a, epi, st);
  if (vpr > 8) return seg_launch<1, 16, 1>(a, epi, st);
  if (vpr > 4) return seg_launch<1, 8, 1>(a, epi, st);
  return seg_launch<1, 4, 1>(a, epi, st);
}

// columns of one pass
static inline int seg_tile(bool vec4) { return vec4 ? 512 : 128; }

static inline SegArgs seg_args(const hb_runs_t* runs, const float* grads, const int64_t* cnt_in, int64_t dim, int mean,
                               const SegPlan& s) {
  SegArgs a;
  a.head = runs->head;
  a.base8 = runs->base8;
  a.perm = runs->perm;
  a.run_start = runs->run_start;
  a.grads = grads;
  a.cnt_in = cnt_in;
  a.n_dev = runs->n_dev;
  a.n = runs->n;
  a.dim = dim;
  a.col0 = 0;
  a.cols = 0;
  a.piece = 0;
  a.mean = mean;
  a.early = 1;
  a.head_part = s.head_part;
  a.tail_part = s.tail_part;
  a.head_cnt = s.head_cnt;
  a.tail_cnt = s.tail_cnt;
  a.done = s.done;
  return a;
}

#endif  // __CUDACC__

}  // namespace hb
