// Sort-once step: the batch of ids is sorted ONCE (radix sort of (id, position)), its runs
// of equal ids are numbered, and everything that the reference does per occurrence is then
// done per distinct id:
//   * hb_runs_build         sort + run heads + class and per-class position of every
//                           distinct id (torch.unique of python/EmbCache/sparse_optim.py:133
//                           and the class lookups of dist_emb.py:174-191, sparse_optim.py:243-259)
//   * hb_lookup_fetch_runs  cache lookup + cached fetch over the sorted batch: consecutive
//                           copies of an id reuse the row already in registers, so a row is read
//                           once per warp that meets it (dist_emb.py:184-243; a DGL sampler hands
//                           the reference unique ids, a raw id stream does not)
//   * hb_runs_miss_list     ids of one class that the cache did not hold, ascending, with
//                           the batch position whose output row holds their embedding
//                           (the uncached cold ids sent to the server, dist_emb.py:218-259)
// The backward aggregation (segsum.cu) and the LRU ageing (index.cu) take the same runs.
#include <type_traits>

#include "a2a.cuh"
#include "compact.cuh"
#include "index.cuh"
#include "maintain.cuh"
#include "runs.cuh"
#include "shard.cuh"
#include "sortcore.cuh"

namespace hb {
int* device_error_word();  // runtime.cu

namespace {

constexpr int kBlock = 256;

// The ids of a batch as sort keys.  Entries at and beyond the device count are left out; entries
// beyond their segment's count sort last.  So does a valid id that is negative or does not fit below
// `sentinel` (2^id_bits - 1): it raises HB_ERR_INVALID in the device status word.
struct IdSource {
  static constexpr bool kSkips = false;
  const int64_t* ids;
  int64_t n;
  const int64_t* n_dev;
  const int64_t* seg_counts;
  uint32_t seg_cap;
  int64_t sentinel;
  int* err;
  int bits;  // stated by the caller
  __host__ __device__ int known_bits() const { return bits; }
  __device__ __forceinline__ int64_t count() const {
    if (!n_dev) return n;
    const int64_t d = *n_dev;
    return d < n ? (d > 0 ? d : 0) : n;
  }
  __device__ __forceinline__ bool fetch(int64_t i, int64_t& id) const {
    if (seg_counts) {
      const uint32_t seg = (uint32_t)i / seg_cap;
      if ((int64_t)((uint32_t)i - seg * seg_cap) >= seg_counts[seg]) return false;
    }
    id = __ldcg(ids + i);  // (as a plain load: 56 bytes of spills in the sort of 65,537 to 303,104 ids)
    return true;
  }
  __device__ __forceinline__ bool accept(int64_t id, unsigned long long& key) const {
    if (id < 0 || id >= sentinel) {
      atomicExch(err, HB_ERR_INVALID);
      return false;
    }
    key = (unsigned long long)id;
    return true;
  }
};

// Runs of equal ids in the sorted order, numbered over all runs and inside the class of their id.  RESOLVE: each
// is looked up where it is written.
template <bool RESOLVE>
struct RunsFinish {
  static constexpr bool kOneEach = RESOLVE;
  const int8_t* table;   // nullable: no classes
  int64_t table_len;
  uint32_t* perm;        // [n]
  uint8_t* head;
  int64_t* uniq;
  int64_t* uniq2;        // nullable second copy (the caller's buffer)
  int64_t* run_start;
  int8_t* dclass;
  int32_t* dpos;
  int64_t* out_ids[3];
  int64_t* num_runs;
  int64_t* num_runs2;    // nullable second copy
  int64_t* class_counts;
  int64_t* class_counts2;
  int32_t* base8;        // [ceil(n / 8)] runs that start before entry 8k
  int64_t* n_valid;      // number of valid entries (read where the input is segmented or large)
  unsigned* zero;        // nullable: words that `resolve` or the next launch needs at zero
  int zero_words;
  struct Nothing {};
  std::conditional_t<RESOLVE, RunsResolve, Nothing> resolve;

  // No runs and no entries: what works on the runs has nothing to do.  The sums go by the entries and do not
  // wait for a device count where the caller has none: they find one run of all entries and no id.
  template <class Ctx>
  __device__ __forceinline__ void give_up(Ctx& ctx, const IdSource& src) const {
    for (int k = threadIdx.x; k < zero_words; k += Ctx::kThreads) zero[k] = 0u;
    for (uint32_t j = ctx.chunk_begin() + threadIdx.x; j < ctx.chunk_end(); j += Ctx::kThreads) {
      perm[j] = j;
      head[j] = j == 0;
      if ((j & 7u) == 0u) base8[j >> 3] = j != 0;
    }
    if (threadIdx.x != 0) return;  // (every CTA writes the same)
    *num_runs = *n_valid = run_start[0] = 0;
    run_start[1] = ctx.count;
    uniq[0] = src.sentinel;
    if (table) {
      dclass[0] = -1;
      dpos[0] = 0;
    }
    if (num_runs2) *num_runs2 = 0;
    for (int c = 0; c < 4; ++c) class_counts[c] = 0;
    for (int c = 0; class_counts2 && c < 3; ++c) class_counts2[c] = 0;
  }

  template <class Ctx>
  __device__ __forceinline__ void run(Ctx& ctx, const IdSource& src) const {
    constexpr int T = Ctx::kThreads, W = T / 32;
    __shared__ int4 s_sum[2 * W + 1];
    __shared__ unsigned long long s_valid;
    const int lane = threadIdx.x & 31;
    for (int k = ctx.rank * T + threadIdx.x; k < zero_words; k += ctx.ctas * T) zero[k] = 0u;
    int ne = ctx.count;
    if (src.seg_counts) {
      // valid entries are scattered over the segments; their number becomes the device count
      if (threadIdx.x == 0) s_valid = 0ull;
      __syncthreads();
      unsigned long long t = 0;
      for (int64_t k = threadIdx.x; k < src.n / src.seg_cap; k += T) {
        const int64_t c = src.seg_counts[k];
        t += (unsigned long long)(c < 0 ? 0 : (c > (int64_t)src.seg_cap ? (int64_t)src.seg_cap : c));
      }
      if (t) atomicAdd(&s_valid, t);
      __syncthreads();
      ne = (int)s_valid;
    }
    const uint32_t begin = ctx.chunk_begin(), end = ctx.chunk_end();
    // id of an entry of the narrow kind (entries that sort last: the sentinel)
    auto narrow_id = [&](uint32_t key) -> int64_t {
      return key == kSortNone && ctx.none ? src.sentinel : (int64_t)key;
    };
    auto wide_id = [&](uint32_t pos) -> int64_t {
      unsigned long long key;
      return sort_load(src, pos, key) ? (int64_t)key : src.sentinel;
    };
    // A thread takes 8 consecutive entries (whole vectors of positions and head flags to
    // write, one entry of base8, no votes), the CTA 8 * T in a strip.
    uint32_t at[8];      // their positions
    uint32_t code = 0u;  // per entry 3 bits: 4 | class (3: none) where a run starts, else 0
    auto classify = [&](uint32_t j0) -> int4 {
      int4 c = make_int4(0, 0, 0, 0);
      code = 0u;
      uint2 e[8];
      e[7] = make_uint2(0u, 0u);
      if (j0 < end) ctx.get8(j0, e);
      uint32_t before = __shfl_up_sync(0xffffffffu, e[7].x, 1);
      if (j0 >= end) return c;
      if (lane == 0 && j0 > 0) before = ctx.get(j0 - 1).x;
      unsigned heads = 0u;
      if (!ctx.wide) {
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          heads |= (unsigned)(j0 + x < (uint32_t)ne && (j0 + x == 0 || e[x].x != before)) << x;
          before = e[x].x;
        }
      } else {
        int64_t was = j0 > 0 ? wide_id(ctx.get(j0 - 1).y) : -1;
#pragma unroll 1
        for (int x = 0; x < 8 && j0 + x < end; ++x) {
          const int64_t id = wide_id(ctx.get(j0 + x).y);
          heads |= (unsigned)(j0 + x < (uint32_t)ne && id != was) << x;
          was = id;
        }
      }
#pragma unroll
      for (int x = 0; x < 8; ++x) at[x] = e[x].y;
      if (!table) {
#pragma unroll
        for (int x = 0; x < 8; ++x) code |= ((heads >> x) & 1u) << (3 * x + 2);
        c.x = __popc(heads);
        return c;
      }
      int8_t cls[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        cls[x] = 3;
        if ((heads >> x) & 1u) {
          const int64_t id = ctx.wide ? wide_id(e[x].y) : narrow_id(e[x].x);
          if (id < table_len) cls[x] = Ctx::kBehindAll ? load_settled(table + id) : table[id];
        }
      }
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        if (!((heads >> x) & 1u)) continue;
        const int k = cls[x] >= 0 && cls[x] <= 2 ? cls[x] : 3;
        code |= (4u | k) << (3 * x);
        c.x += k == 0;
        c.y += k == 1;
        c.z += k == 2;
        c.w += k == 3;
      }
      return c;
    };
    auto put_entries = [&](uint32_t j0) {
      if (j0 >= end) return;
      if (j0 + 8 <= end) {
        uint4* p = reinterpret_cast<uint4*>(perm + j0);
        p[0] = make_uint4(at[0], at[1], at[2], at[3]);
        p[1] = make_uint4(at[4], at[5], at[6], at[7]);
      } else {
#pragma unroll
        for (int x = 0; x < 8; ++x)
          if (j0 + x < end) perm[j0 + x] = at[x];
      }
      // one byte per entry (the allocation holds whole groups of 8)
      auto flag = [&](int x) -> uint32_t { return (code >> (3 * x + 2)) & 1u; };
      const uint32_t lo = flag(0) | (flag(1) << 8) | (flag(2) << 16) | (flag(3) << 24);
      const uint32_t hi = flag(4) | (flag(5) << 8) | (flag(6) << 16) | (flag(7) << 24);
      *reinterpret_cast<uint2*>(head + j0) = make_uint2(lo, hi);
    };
    // a thread's counts -> those of the threads ahead in its warp and of the whole warp
    auto scan_warp = [&](const int4& c, int4& total) -> int4 {
      const unsigned long long v = (unsigned long long)(uint32_t)(c.x | (c.y << 16)) | ((unsigned long long)(uint32_t)(c.z | (c.w << 16)) << 32);
      unsigned long long inc = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      const unsigned long long t = __shfl_sync(0xffffffffu, inc, 31);
      total = make_int4((int)(t & 0xffff), (int)((t >> 16) & 0xffff), (int)((t >> 32) & 0xffff), (int)(t >> 48));
      inc -= v;
      return make_int4((int)(inc & 0xffff), (int)((inc >> 16) & 0xffff), (int)((inc >> 32) & 0xffff), (int)(inc >> 48));
    };
    uint32_t kept = 0u;  // the codes of the first of two strips
    // (stores ahead of the barrier are what it waits for; that a kernel has them behind it, and then one strip, is known
    // when it is compiled: 512 ids with their classes 10.8 -> 10.3 us, 8,192 17.3 -> 16.8)
    constexpr bool late = Ctx::kStoresLate;
    const int strips = late ? (int)(end > begin) : (int)((end - begin + 8 * T - 1) / (8 * T));
    int4 mine = make_int4(0, 0, 0, 0), lanes = mine, warps, cta, ahead, all;
#pragma unroll 1
    for (int q = 0; q < strips; ++q) {
      const uint32_t j0 = begin + q * (8 * T) + threadIdx.x * 8;
      const int4 c = classify(j0);
      if (!late) put_entries(j0);
      int4 total;
      lanes = scan_warp(c, total);
      mine.x += total.x; mine.y += total.y; mine.z += total.z; mine.w += total.w;
      if (q == 0) kept = code;
    }
    sort_warp_sums<W>(mine, s_sum, warps, cta);
    if (!ctx.prefix(cta, ahead, all)) return give_up(ctx, src);
    if (late) put_entries(begin + threadIdx.x * 8);
#pragma unroll 1
    for (int q = 0; q < strips; ++q) {
      const uint32_t strip = begin + q * (8 * T);
      const uint32_t j0 = strip + threadIdx.x * 8;
      if (strips > 1) {
        int4 total, c = make_int4(0, 0, 0, 0);
        if (strips > 2) {
          c = classify(j0);
        } else {
          const uint32_t last = code;  // strip 1 was classified last: its codes stay for the next turn
          if (q == 0) code = kept;
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const uint32_t v = (code >> (3 * x)) & 7u;
            c.x += v == 4u;
            c.y += v == 5u;
            c.z += v == 6u;
            c.w += v == 7u;
          }
          if (q == 0) kept = last;
        }
        lanes = scan_warp(c, total);
        __syncthreads();
        sort_warp_sums<W>(total, s_sum, warps, cta);
      }
      // The runs of the strip as a list in shared memory, so that what is written per run leaves in
      // whole sectors: 13 bits place in the strip, 2 class, 14 number inside the class and strip.
      int4 run = make_int4(warps.x + lanes.x, warps.y + lanes.y, warps.z + lanes.z, warps.w + lanes.w);
      const int before = ahead.x + ahead.y + ahead.z + ahead.w;
      if (j0 < end) base8[j0 >> 3] = before + run.x + run.y + run.z + run.w;
      if (code) {
        int at = run.x + run.y + run.z + run.w;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const uint32_t c = (code >> (3 * x)) & 7u;
          if (!c) continue;
          const uint32_t k = c & 3u;
          const int pos = k == 0 ? run.x : (k == 1 ? run.y : (k == 2 ? run.z : run.w));
          ctx.scratch[at++] = (threadIdx.x * 8 + x) | (k << 13) | ((uint32_t)pos << 15);
          run.x += k == 0;
          run.y += k == 1;
          run.z += k == 2;
          run.w += k == 3;
        }
      }
      __syncthreads();
      const int runs = cta.x + cta.y + cta.z + cta.w;
      auto put = [&](int r, int64_t& id, bool& cold) {
        const uint32_t w = ctx.scratch[r];
        const uint32_t j = strip + (w & 8191u);
        const uint2 e = ctx.get(j);
        id = ctx.wide ? wide_id(e.y) : narrow_id(e.x);
        const int u = before + r;
        uniq[u] = id;
        if (uniq2) uniq2[u] = id;
        run_start[u] = j;
        if (table) {
          const int k = (int)(w >> 13) & 3;
          const int pos = (int)(w >> 15) + (k == 0 ? ahead.x : (k == 1 ? ahead.y : (k == 2 ? ahead.z : ahead.w)));
          dclass[u] = k < 3 ? (int8_t)k : (int8_t)-1;
          dpos[u] = pos;
          int64_t* to = k == 0 ? out_ids[0] : (k == 1 ? out_ids[1] : (k == 2 ? out_ids[2] : nullptr));
          if (to) to[pos] = id;
          cold = k == 2;
        }
      };
      if constexpr (RESOLVE) {
#pragma unroll 1
        for (int r = threadIdx.x; r - lane < runs; r += T) {  // whole warps
          int64_t id = -1;
          bool cold = false;
          if (r < runs) put(r, id, cold);
          resolve_run(resolve, before + r, r < runs, id, cold);
        }
      } else {
#pragma unroll 2
        for (int r = threadIdx.x; r < runs; r += T) {
          int64_t id;
          bool cold;
          put(r, id, cold);
        }
      }
      if (strips > 1) __syncthreads();
      if (strips == 2) code = kept;
      ahead.x += cta.x; ahead.y += cta.y; ahead.z += cta.z; ahead.w += cta.w;
    }
    if (ctx.rank == 0 && threadIdx.x == 0) {
      const int64_t u = (int64_t)all.x + all.y + all.z + all.w;
      *num_runs = u;
      if (num_runs2) *num_runs2 = u;
      run_start[u] = ne;
      *n_valid = ne;
      class_counts[0] = all.x; class_counts[1] = all.y; class_counts[2] = all.z; class_counts[3] = all.w;
      if (class_counts2) { class_counts2[0] = all.x; class_counts2[1] = all.y; class_counts2[2] = all.z; }
    }
  }
};

// ---- forward: lookup + fetch over the sorted batch -----------------------------------------
// RESOLVE works per distinct id (one lane per run): the index probe, the slot of the run, and
// where the row of the run is to be read from -- the cache row, the row of the table on this
// GPU, or, for a row that lives on ANOTHER GPU, its place in a staging buffer on this GPU; such
// runs go on a list.  STAGE (sharded tables only) copies the listed rows from their owners, so
// that every remote row crosses NVLink once per step however often its id occurs in the batch
// (a row read again by every warp that meets the id, from seven GPUs at once, serialises on one
// L2 slice of its owner).  EXPAND works per entry of the sorted batch: the row goes to the
// entry's batch position; entries of one run inside a warp take the registers of the first.
struct RowSource {
  const char* backing;  // one table on this GPU, or null
  int64_t backing_rows;
  ShardView shards;     // used when PEER
  int rank;             // whose shard is local (PEER)
  char* stage;          // [stage_cap][row_bytes] copies of remote rows, by run (PEER)
  int64_t stage_cap;
  int32_t* remote_runs;            // runs whose row STAGE has to copy, in any order (PEER)
  unsigned long long* remote_count;  // [1], zero before RESOLVE
  // when the OWNERS deliver the remote rows (hb_runs_resolve_requests): a remote run becomes the
  // request (id, run) -- the run is also the row of this GPU's stage that the owner fills --
  // stored straight into this rank's slab of the owner's receive area
  const hb_a2a::Dest* req_dest;
  unsigned long long* req_counts;  // [world] requests so far per owner, zero before RESOLVE
  int64_t req_cap;                 // requests one owner's slab takes from this rank
};

template <bool PEER>
__device__ __forceinline__ uint4 load_row16(const uint4* p) {
  if (PEER) return *p;  // may be a peer GPU's memory that its owner rewrites between steps
  return load_settled(p);  // (the launch before it looks the rows up)
}

// run_src[u]: address of the run's row (16-byte aligned, 0 = none) | 1 when it is a cache row
template <int MODE, bool PEER>
__global__ void __launch_bounds__(kBlock) runs_resolve_kernel(
    IndexView v, hb_runs_t r, RowSource rs, const char* __restrict__ cache_rows, int64_t row_bytes,
    int vb, unsigned long long* __restrict__ run_src, int64_t* __restrict__ run_slots,
    int* __restrict__ err) {
  __shared__ int64_t s_top[MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  const int64_t U = *r.num_runs;
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t limit = PEER ? rs.shards.num_rows : rs.backing_rows;
  for (int64_t u0 = warp * 32; u0 < U; u0 += nwarps * 32) {
    const int64_t u = u0 + lane;
    const bool valid = u < U;
    const int64_t id = valid ? __ldg(r.uniq_ids + u) : -1;
    const int64_t slot = warp_lookup<MODE>(v, s_top, id);
    const char* src = nullptr;
    const char* remote = nullptr;  // to be copied to the stage
    if (slot >= 0) {
      src = cache_rows + slot * row_bytes;
    } else if (valid && id < limit) {
      if (PEER) {
        const char* row = shard_row(rs.shards, id, row_bytes);
        const bool mine = rs.shards.world == 1 || mod_nonneg(id, rs.shards.world) == rs.rank;
        if (mine || u >= rs.stage_cap) {
          src = row;  // local shard, or no room in the stage: EXPAND reads the owner's memory itself
        } else {
          remote = row;
          src = rs.stage + u * row_bytes;
        }
      } else {
        src = rs.backing ? rs.backing + id * row_bytes : nullptr;
      }
    } else if (valid && (PEER || rs.backing)) {
      atomicExch(err, HB_ERR_INVALID);  // no such row: the output rows of the run stay as they were
    }
    if (valid) {
      run_src[u] = (unsigned long long)src | (slot >= 0 ? 1ull : 0ull);
      if (run_slots) run_slots[u] = slot;
    }
    if (PEER) {
      // remote runs go on a list; STAGE copies their rows with every row in flight at once (the
      // copy is bound by round trips over NVLink, which a kernel that also probes the index
      // cannot keep enough of in flight)
      const unsigned todo = __ballot_sync(0xffffffffu, remote != nullptr);
      if (todo && rs.req_dest) {
        if (remote) {
          // one counter per owner: the lanes that ask the same owner take consecutive places
          const int owner = (int)mod_nonneg(id, rs.shards.world);
          const unsigned same = __match_any_sync(todo, owner);
          const int leader = __ffs(same) - 1;
          unsigned long long at = 0;
          if (lane == leader) at = atomicAdd(rs.req_counts + owner, (unsigned long long)__popc(same));
          at = __shfl_sync(same, at, leader);
          const int64_t k = (int64_t)at + __popc(same & ((1u << lane) - 1u));
          if (k < rs.req_cap) {
            const int64_t slot = (int64_t)rs.rank * rs.req_cap + k;  // my slab in the owner's area
            rs.req_dest->ids[owner][slot] = id;
            rs.req_dest->cnt[owner][slot] = u;
          } else {
            atomicExch(err, HB_ERR_CAPACITY);  // the row is not delivered: the stage keeps what it held
          }
        }
      } else if (todo) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(rs.remote_count, (unsigned long long)__popc(todo));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (remote) rs.remote_runs[at + __popc(todo & ((1u << lane) - 1u))] = (int32_t)u;
      }
    }
  }
}

// STAGE: the rows of the listed runs, from their owners' shards into this GPU's stage.  One
// warp per row and step, 4 rows in flight per warp, 32 warps per SM: some 19,000 rows are on
// their way at once, several times what the links need to run at their bandwidth.
__global__ void __launch_bounds__(kBlock, 4) runs_stage_kernel(hb_runs_t r, RowSource rs, int64_t row_bytes, int vb) {
  const int64_t cnt = (int64_t)*rs.remote_count;
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  constexpr int kFly = 4;
  for (int64_t i0 = warp * kFly; i0 < cnt; i0 += nwarps * kFly) {
    const char* from[kFly];
    char* to[kFly];
#pragma unroll
    for (int x = 0; x < kFly; ++x) {
      from[x] = nullptr;
      to[x] = nullptr;
      if (i0 + x < cnt) {
        // every rank starts at another place of its list: the lists of the ranks hold much the same
        // popular ids in much the same order, and readers that walk an owner's rows in step with
        // each other queue on the same lines
        int64_t at = i0 + x + (cnt / rs.shards.world) * rs.rank;
        if (at >= cnt) at -= cnt;
        const int64_t u = rs.remote_runs[at];
        from[x] = shard_row(rs.shards, __ldg(r.uniq_ids + u), row_bytes);
        to[x] = rs.stage + u * row_bytes;
      }
    }
    if (vb == 16) {
      for (int64_t k = lane; k < (row_bytes >> 4); k += 32) {
        uint4 val[kFly];
#pragma unroll
        for (int x = 0; x < kFly; ++x)
          if (from[x]) val[x] = *(reinterpret_cast<const uint4*>(from[x]) + k);
#pragma unroll
        for (int x = 0; x < kFly; ++x)
          if (from[x]) *(reinterpret_cast<uint4*>(to[x]) + k) = val[x];
      }
    } else {
      for (int x = 0; x < kFly; ++x) {
        if (!from[x]) continue;
        for (int64_t k = lane; k < row_bytes; k += 32) to[x][k] = from[x][k];
      }
    }
  }
}

// the run an entry of the sorted batch belongs to: runs that start before its group of 8
// entries (base8) + the heads inside the group up to the entry
__device__ __forceinline__ int64_t run_of_entry(const hb_runs_t& r, int64_t j) {
  const unsigned long long flags = *reinterpret_cast<const unsigned long long*>(r.head + (j & ~(int64_t)7));
  const int k = (int)(j & 7);
  const unsigned long long mask = k == 7 ? ~0ull : ((1ull << (8 * (k + 1))) - 1ull);
  return (int64_t)r.base8[j >> 3] + __popcll(flags & mask) - 1;
}

// The id of every sorted entry; entries that take no part hold the sentinel.  perm (nullable): positions
// at and beyond the device count follow in order.
template <typename K>
__global__ void __launch_bounds__(kBlock) runs_keys_kernel(hb_runs_t r, int64_t sentinel, K* __restrict__ keys,
                                                           uint32_t* __restrict__ perm) {
  const int64_t n = runs_valid_entries(r);
  for (int64_t j = blockIdx.x * (int64_t)kBlock + threadIdx.x; j < r.n; j += (int64_t)gridDim.x * kBlock) {
    keys[j] = (K)(j < n ? __ldg(r.uniq_ids + run_of_entry(r, j)) : sentinel);
    if (perm && j >= n) perm[j] = (uint32_t)j;
  }
}

// RB: 512 = rows of exactly 512 bytes (128 fp32: the address arithmetic folds, no lane is idle);
// 16 = any multiple of 16 bytes; 0 = words or bytes.  PEER: a source may be another GPU's memory
// (runs that found no room in the stage), so rows are read with plain loads.
// MAINTAIN: blocks that bring the index up to date meanwhile, the first of the launch or spread over it (a chain of
// dependent reads beside a stream of rows: a second launch of it costs more than it takes).
// FULL: 32 entries a warp and round, known here: the batches of rows in flight unroll over a fixed range, and
// rows of 512 bytes take no spills at 64 registers (with a number known at run time 44 to 60 bytes: 2,000,000
// distinct ids 0.376 -> 0.441 ms).  The other form is for lists that do not fill the GPU.
template <bool PEER, int RB, bool MAINTAIN, bool FULL>
__global__ void __launch_bounds__(kBlock, RB == 512 ? 4 : 3) runs_expand_kernel(
    hb_runs_t r, const unsigned long long* run_src, const int64_t* run_slots, int64_t row_bytes_arg, int vb, char* out,
    int64_t* locs, uint8_t* found, int per_arg, Maintain duty) {
  begin_after_previous();
  const int per = FULL ? 32 : per_arg;
  int block = blockIdx.x, blocks = gridDim.x;
  if (MAINTAIN) {
    int before = block < duty.blocks ? block : duty.blocks, upto = block < duty.blocks ? block + 1 : duty.blocks;
    if (duty.spread) {
      before = (int)((unsigned)block * (unsigned)duty.blocks / (unsigned)blocks);
      upto = (int)((unsigned)(block + 1) * (unsigned)duty.blocks / (unsigned)blocks);
    }
    if (upto != before) {
      duty.template run<kBlock>(before);
      return;
    }
    block -= before;
    blocks -= duty.blocks;
  }
  constexpr bool V16 = RB != 0;
  const int64_t row_bytes = RB == 512 ? (int64_t)512 : row_bytes_arg;
  const int64_t n = runs_valid_entries(r);
  const int lane = lane_id();
  const int64_t warp = (block * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t stride = (((int64_t)blocks * blockDim.x) >> 5) * per;
  int64_t base = warp * per;
  uint32_t pos_next = 0;
  int64_t run_next = -1;
  if (lane < per && base + lane < n) {
    pos_next = r.perm[base + lane];
    run_next = run_of_entry(r, base + lane);
  }
  for (; base < n; base += stride) {
    const bool valid = lane < per && base + lane < n;
    const uint32_t pos = pos_next;
    const int64_t u = valid ? run_next : -1;
    if (lane < per && base + stride + lane < n) {
      pos_next = r.perm[base + stride + lane];
      run_next = run_of_entry(r, base + stride + lane);
    }
    const int64_t prev = __shfl_up_sync(0xffffffffu, u, 1);
    const unsigned fresh = __ballot_sync(0xffffffffu, lane == 0 || u != prev);
    const unsigned long long word = valid ? run_src[u] : 0ull;
    const unsigned long long src_bits = word & ~1ull;
    if (valid) {
      if (found) found[pos] = (uint8_t)(word & 1ull);
      if (locs) locs[pos] = run_slots[u];  // 8 bytes scattered over the batch: costly
    }
    const unsigned have = __ballot_sync(0xffffffffu, src_bits != 0ull);
    if (V16) {
      const int64_t vpr = row_bytes >> 4;
      if (RB == 512 || vpr <= 32) {
        const bool on = RB == 512 || lane < vpr;
        uint4 last = make_uint4(0, 0, 0, 0);
        constexpr int kFly = RB == 512 ? 8 : 4;  // rows whose loads are in flight together
        for (int q0 = 0; q0 < per; q0 += kFly) {
          if (((have >> q0) & ((1u << kFly) - 1u)) == 0u) continue;
          uint4 val[kFly];
          uint32_t pq[kFly];
#pragma unroll
          for (int x = 0; x < kFly; ++x) {
            const int q = q0 + x;
            const unsigned long long sb = __shfl_sync(0xffffffffu, src_bits, q);
            pq[x] = __shfl_sync(0xffffffffu, pos, q);
            if (((have & fresh) >> q) & 1u)
              if (on) val[x] = load_row16<PEER>(reinterpret_cast<const uint4*>(sb) + lane);
          }
#pragma unroll
          for (int x = 0; x < kFly; ++x) {
            const int q = q0 + x;
            if (!((have >> q) & 1u)) continue;
            if (!((fresh >> q) & 1u)) val[x] = last;
            last = val[x];
            if (on) __stcs(reinterpret_cast<uint4*>(out + (int64_t)pq[x] * row_bytes) + lane, val[x]);
          }
        }
      } else {
        for (int q0 = 0; q0 < per; q0 += 4) {
          if (((have >> q0) & 0xfu) == 0u) continue;
          const uint4* sp[4];
          uint4* dp[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const int q = q0 + x;
            const unsigned long long sb = __shfl_sync(0xffffffffu, src_bits, q);
            const uint32_t pq = __shfl_sync(0xffffffffu, pos, q);
            sp[x] = ((have >> q) & 1u) ? reinterpret_cast<const uint4*>(sb) : nullptr;
            dp[x] = reinterpret_cast<uint4*>(out + (int64_t)pq * row_bytes);
          }
          for (int64_t k = lane; k < vpr; k += 32) {
            uint4 val[4];
#pragma unroll
            for (int x = 0; x < 4; ++x)
              if (sp[x]) val[x] = load_row16<PEER>(sp[x] + k);
#pragma unroll
            for (int x = 0; x < 4; ++x)
              if (sp[x]) __stcs(dp[x] + k, val[x]);
          }
        }
      }
    } else {
      // rows that are not a multiple of 16 bytes (or unaligned buffers): words or bytes
      for (int q = 0; q < per; ++q) {
        const unsigned long long sb = __shfl_sync(0xffffffffu, src_bits, q);
        const uint32_t pq = __shfl_sync(0xffffffffu, pos, q);
        if (!((have >> q) & 1u)) continue;
        char* d = out + (int64_t)pq * row_bytes;
        if (vb == 4) {
          const uint32_t* s4 = reinterpret_cast<const uint32_t*>(sb);
          for (int64_t k = lane; k < (row_bytes >> 2); k += 32) reinterpret_cast<uint32_t*>(d)[k] = s4[k];
        } else {
          const char* s1 = reinterpret_cast<const char*>(sb);
          for (int64_t k = lane; k < row_bytes; k += 32) d[k] = s1[k];
        }
      }
    }
  }
}

// ---- ids of one class that missed the cache -----------------------------------------------
struct MissPolicy {
  hb_runs_t r;
  const int64_t* locs;   // slot per batch position (kind 0), per sorted entry (1) or per run (2)
  int locs_kind;
  int want_class;        // < 0: every class
  int64_t cap;
  int64_t* miss_ids;     // [cap], filled from entry 0
  int64_t* miss_src;     // [cap] batch position whose output row holds the embedding
  int64_t* miss_count;
  __device__ __forceinline__ int classify(int64_t u) const {
    if (u >= *r.num_runs) return -1;
    if (want_class >= 0 && (!r.dclass || r.dclass[u] != want_class)) return -1;
    const int64_t j = r.run_start[u];
    const int64_t at = locs_kind == 2 ? u : (locs_kind == 1 ? j : (int64_t)r.perm[j]);
    return locs[at] < 0 ? 0 : -1;
  }
  __device__ __forceinline__ void emit(int64_t u, int, const int4& before) const {
    if (before.x >= cap) return;
    miss_ids[before.x] = r.uniq_ids[u];
    miss_src[before.x] = (int64_t)r.perm[r.run_start[u]];
  }
  __device__ __forceinline__ void finish(const int4& tot) const {
    *miss_count = tot.x < cap ? tot.x : cap;
  }
};

__global__ void fill_i64_kernel(int64_t* p, int64_t n, int64_t v) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

}  // namespace

RunsPlan make_runs_plan(void* ws, int64_t n, bool keys) {
  RunsPlan s;
  Carver cv(ws ? ws : (void*)256);  // a null workspace still yields the sizes
  const int64_t m = n > 0 ? n : 1;
  s.perm = cv.take<uint32_t>(m);
  s.sort_ws = cv.take<char>(sort_grid_bytes(m));
  s.run_start = cv.take<int64_t>(m + 1);
  s.head = cv.take<uint8_t>(m + 8);
  s.n_valid = cv.take<int64_t>(1);
  s.num_runs = cv.take<int64_t>(1);
  s.class_counts = cv.take<int64_t>(4);
  s.dclass = cv.take<int8_t>(m + 1);
  s.dpos = cv.take<int32_t>(m + 1);
  s.uniq = cv.take<int64_t>(m + 1);
  s.base8 = cv.take<int32_t>(m / 8 + 2);
  s.keys = keys ? cv.take<int64_t>(m) : nullptr;
  s.total = cv.used() + 256;
  return s;
}

}  // namespace hb

using namespace hb;

extern "C" {

size_t hb_runs_workspace_bytes(int64_t n) { return make_runs_plan(nullptr, n, true).total; }

int hb_runs_build(const int64_t* ids, int64_t n, const int64_t* n_dev, const int64_t* seg_counts,
                  int64_t seg_cap, int id_bits, const int8_t* class_table, int64_t table_len,
                  int64_t* const* class_ids_out, int64_t* class_counts_out, int64_t* uniq_ids_out,
                  int64_t* num_unique_out, void* workspace, size_t workspace_bytes,
                  hb_runs_t* runs_out, hb_stream_t stream) {
  if (workspace && workspace_bytes < hb_runs_workspace_bytes(n)) workspace = nullptr;  // (runs_build says what is missing)
  const int rc = runs_build(ids, n, n_dev, seg_counts, seg_cap, id_bits, class_table, table_len, class_ids_out,
                            class_counts_out, uniq_ids_out, num_unique_out, nullptr, 0, workspace, workspace_bytes,
                            runs_out, (cudaStream_t)stream);
  return rc != HB_OK ? rc : runs_keys(seg_counts, id_bits, workspace, runs_out, (cudaStream_t)stream);
}

}  // extern "C"

// what stands for an entry without a valid id: above every other
static int64_t runs_sentinel(int id_bits) { return id_bits >= 63 ? INT64_MAX : (((int64_t)1 << id_bits) - 1); }

int hb::runs_keys(const int64_t* seg_counts, int id_bits, void* workspace, hb_runs_t* runs, cudaStream_t st) {
  runs->keys = nullptr;
  runs->key_bytes = 0;
  if (runs->n == 0) return HB_OK;
  const RunsPlan s = make_runs_plan(workspace, runs->n, true);
  int64_t blocks = ceil_div(runs->n, kBlock);
  if (blocks > (int64_t)sm_count() * 16) blocks = (int64_t)sm_count() * 16;
  uint32_t* rest = seg_counts ? nullptr : s.perm;
  if (id_bits <= 32)
    HB_LAUNCH(runs_keys_kernel<uint32_t>, (int)blocks, kBlock, 0, st, *runs, runs_sentinel(id_bits), (uint32_t*)s.keys, rest);
  else
    HB_LAUNCH(runs_keys_kernel<int64_t>, (int)blocks, kBlock, 0, st, *runs, runs_sentinel(id_bits), (int64_t*)s.keys, rest);
  runs->keys = s.keys;
  runs->key_bytes = id_bits <= 32 ? 4 : 8;
  return HB_OK;
}

int hb::runs_build(const int64_t* ids, int64_t n, const int64_t* n_dev, const int64_t* seg_counts, int64_t seg_cap,
                   int id_bits, const int8_t* class_table, int64_t table_len, int64_t* const* class_ids_out,
                   int64_t* class_counts_out, int64_t* uniq_ids_out, int64_t* num_unique_out, unsigned* zero,
                   int64_t zero_words, void* workspace, size_t workspace_bytes, hb_runs_t* runs_out,
                   cudaStream_t st, const RunsResolve* resolve) {
  HB_CHECK_ARG(runs_out != nullptr, "hb_runs_build: runs_out is null");
  HB_CHECK_ARG(n >= 0 && n < ((int64_t)1 << 31), "hb_runs_build: n out of range");
  HB_CHECK_ARG(n == 0 || ids, "hb_runs_build: null ids");
  HB_CHECK_ARG(id_bits >= 1 && id_bits <= 64, "hb_runs_build: id_bits must be in [1, 64]");
  HB_CHECK_ARG(!seg_counts || (seg_cap > 0 && n % seg_cap == 0),
               "hb_runs_build: a segmented input holds whole segments of seg_cap entries");
  HB_CHECK_ARG(!class_table || table_len > 0, "hb_runs_build: a class table needs its length");
  RunsPlan s = make_runs_plan(workspace, n, false);
  if (!workspace || workspace_bytes < s.total) {
    set_error("hb_runs_build: workspace of %zu bytes needed, %zu given", hb_runs_workspace_bytes(n), workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  memset(runs_out, 0, sizeof(*runs_out));
  runs_out->n = n;
  runs_out->num_runs = s.num_runs;
  runs_out->class_counts = s.class_counts;
  runs_out->run_start = s.run_start;
  runs_out->head = s.head;
  runs_out->uniq_ids = s.uniq;
  runs_out->base8 = s.base8;
  runs_out->dclass = class_table ? s.dclass : nullptr;
  runs_out->dpos = class_table ? s.dpos : nullptr;
  if (n == 0) {
    HB_CUDA(cudaMemsetAsync(s.num_runs, 0, sizeof(int64_t), st));
    HB_CUDA(cudaMemsetAsync(s.class_counts, 0, 4 * sizeof(int64_t), st));
    HB_CUDA(cudaMemsetAsync(s.run_start, 0, sizeof(int64_t), st));
    if (num_unique_out) HB_CUDA(cudaMemsetAsync(num_unique_out, 0, sizeof(int64_t), st));
    if (class_counts_out) HB_CUDA(cudaMemsetAsync(class_counts_out, 0, 3 * sizeof(int64_t), st));
    return HB_OK;
  }
  // (a grid whose barrier runs out leaves no entries)
  runs_out->n_dev = seg_counts || n > kSortClusterMax ? s.n_valid : n_dev;
  const int64_t sentinel = runs_sentinel(id_bits);
  runs_out->perm = s.perm;
  IdSource src{ids, n, seg_counts ? nullptr : n_dev, seg_counts, (uint32_t)(seg_counts ? seg_cap : 1), sentinel,
               device_error_word(), id_bits};
  static_assert(kResolvedMax <= kSortOneEach, "one run per thread");
  auto run = [&](auto fin) -> int {
    fin.table = class_table;
    fin.table_len = table_len;
    fin.perm = s.perm;
    fin.head = s.head;
    fin.uniq = s.uniq;
    fin.uniq2 = uniq_ids_out;
    fin.run_start = s.run_start;
    fin.dclass = s.dclass;
    fin.dpos = s.dpos;
    for (int c = 0; c < 3; ++c) fin.out_ids[c] = class_ids_out ? class_ids_out[c] : nullptr;
    fin.num_runs = s.num_runs;
    fin.num_runs2 = num_unique_out;
    fin.class_counts = s.class_counts;
    fin.class_counts2 = class_counts_out;
    fin.base8 = s.base8;
    fin.n_valid = s.n_valid;
    fin.zero = zero;
    fin.zero_words = (int)zero_words;
    if constexpr (decltype(fin)::kOneEach) fin.resolve = *resolve;
    return sort_run(src, fin, n, s.sort_ws, st);
  };
  return resolve ? run(RunsFinish<true>{}) : run(RunsFinish<false>{});
}

extern "C" {

namespace {
// scratch of hb_lookup_fetch_runs: where every run's row is read from, the slot of every run
// when the caller does not ask for it, and (sharded table) the copies of the remote rows
struct FetchPlan {
  unsigned long long* run_src;
  int64_t* run_slots;
  char* stage;
  int64_t stage_cap;
  int32_t* remote_runs;
  unsigned long long* remote_count;
  unsigned long long* req_counts;  // [64]
  size_t total;
};
constexpr int64_t kStageMaxBytes = (int64_t)1 << 30;  // at most 1 GiB of staged remote rows

FetchPlan make_fetch_plan(void* ws, int64_t n, int64_t row_bytes, bool sharded) {
  FetchPlan f;
  Carver cv(ws ? ws : (void*)256);
  const int64_t m = n > 0 ? n : 1;
  f.run_src = cv.take<unsigned long long>(m);
  f.run_slots = cv.take<int64_t>(m);
  f.req_counts = cv.take<unsigned long long>(64);
  f.stage_cap = 0;
  f.stage = nullptr;
  f.remote_runs = nullptr;
  f.remote_count = nullptr;
  if (sharded) {
    f.stage_cap = kStageMaxBytes / row_bytes < m ? kStageMaxBytes / row_bytes : m;
    f.stage = cv.take<char>((size_t)f.stage_cap * row_bytes);
    f.remote_runs = cv.take<int32_t>(m);
    f.remote_count = cv.take<unsigned long long>(2);
  }
  f.total = cv.used() + 256;
  return f;
}
// Who brings the remote rows: nobody (one table on this GPU), this GPU (STAGE reads the owners'
// shards), or the owners (`dv`: RESOLVE lists (id, run) requests, the owners store the rows into
// dv->stage, which they have mapped, before EXPAND runs).
struct Delivery {
  char* stage;
  int64_t stage_cap;
  hb_a2a* requests;  // the exchange that carries the requests (null: expansion only)
  int* parity_out;   // which of its receive areas this call filled
  bool peer_sources; // expansion only: a run's row may lie in another GPU's memory (plain loads)
};

int fetch_runs_impl(hb_index_t* h, const hb_runs_t* runs, const void* cache_rows, const void* backing_rows,
                    int64_t backing_num_rows, hb_peer_table_t* table, int64_t row_bytes, void* out_rows,
                    int64_t* locs, uint8_t* found, int64_t* run_slots, int mode, void* workspace,
                    size_t workspace_bytes, hb_stream_t stream, const Delivery* dv, bool resolve, bool expand) {
  HB_CHECK_ARG((h || !resolve) && runs, "hb_lookup_fetch_runs: null argument");
  HB_CHECK_ARG(row_bytes > 0, "hb_lookup_fetch_runs: bad row size");
  HB_CHECK_ARG(runs->n == 0 || ((cache_rows || !resolve) && runs->perm && runs->head && runs->base8 &&
                                runs->uniq_ids),
               "hb_lookup_fetch_runs: null argument");
  HB_CHECK_ARG(mode == HB_LOOKUP_SETASSOC || mode == HB_LOOKUP_SORTED,
               "hb_lookup_fetch_runs: unknown mode %d", mode);
  HB_CHECK_ARG(!(table && backing_rows), "hb_lookup_fetch_runs: give a backing table or a sharded one");
  HB_CHECK_ARG(!table || table->row_bytes == row_bytes, "hb_lookup_fetch_runs: row size differs from the table's");
  HB_CHECK_ARG(!backing_rows || backing_num_rows > 0, "hb_lookup_fetch_runs: a backing table needs its row count");
  cudaStream_t st = (cudaStream_t)stream;
  FetchPlan f0 = make_fetch_plan(workspace, runs->n, row_bytes, false);
  if (resolve && dv && dv->requests) {
    // also with an empty batch: the owners read this rank's counts after the fence
    if (!workspace || workspace_bytes < f0.total) {
      set_error("hb_runs_resolve_requests: workspace of %zu bytes needed, %zu given", f0.total, workspace_bytes);
      return HB_ERR_WORKSPACE;
    }
    HB_CUDA(cudaMemsetAsync(f0.req_counts, 0, 64 * sizeof(unsigned long long), st));
  }
  if (runs->n == 0) {
    if (resolve && dv && dv->requests) {
      const hb_a2a::Dest* dest;
      int rc = a2a_direct_begin(dv->requests, &dest, dv->parity_out);
      if (rc != HB_OK) return rc;
      return a2a_direct_publish(dv->requests, *dv->parity_out, f0.req_counts, st);
    }
    return HB_OK;
  }
  const bool sharded = !dv && table != nullptr && table->world > 1;  // this GPU copies the remote rows
  FetchPlan f = make_fetch_plan(workspace, runs->n, row_bytes, sharded);
  if (!workspace || workspace_bytes < f.total) {
    set_error("hb_lookup_fetch_runs: workspace of %zu bytes needed, %zu given", f.total, workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  if (resolve && mode == HB_LOOKUP_SORTED && h->sorted_stale) {
    int rc = hb_index_build_sorted(h, stream);
    if (rc != HB_OK) return rc;
  }
  RowSource rs;
  memset(&rs, 0, sizeof(rs));
  rs.backing = (const char*)backing_rows;
  rs.backing_rows = backing_rows ? backing_num_rows : 0;
  rs.stage = f.stage;
  rs.stage_cap = f.stage_cap;
  rs.remote_runs = f.remote_runs;
  rs.remote_count = f.remote_count;
  if (dv) {
    rs.stage = dv->stage;
    rs.stage_cap = dv->stage_cap;
    if (resolve && dv->requests) {
      HB_CHECK_ARG(dv->requests->world == table->world && dv->requests->rank == table->rank,
                   "hb_runs_resolve_requests: the exchange and the table belong to different groups");
      int rc = a2a_direct_begin(dv->requests, &rs.req_dest, dv->parity_out);
      if (rc != HB_OK) return rc;
      rs.req_counts = f.req_counts;
      rs.req_cap = dv->requests->cap;
    }
  }
  if (table) {
    int rc = make_shard_view(table, &rs.shards);
    if (rc != HB_OK) return rc;
    rs.rank = table->rank;
  }
  uintptr_t bits = (uintptr_t)row_bytes | (uintptr_t)cache_rows | (uintptr_t)out_rows | (uintptr_t)backing_rows |
                   (uintptr_t)(dv ? dv->stage : nullptr);
  HB_CHECK_ARG((bits & 1) == 0, "hb_lookup_fetch_runs: rows must start at even addresses");
  const bool v16 = (bits & 15) == 0;  // shards come from cudaMalloc and hold whole rows
  const int vb = v16 ? 16 : ((bits & 3) == 0 ? 4 : 1);
  int* err = device_error_word();
  int64_t* slots = run_slots ? run_slots : f.run_slots;
  if (resolve && sharded) HB_CUDA(cudaMemsetAsync(rs.remote_count, 0, sizeof(unsigned long long), st));
  if (resolve) {
    int64_t blocks = ceil_div(ceil_div(runs->n, 32) * 32, kBlock);  // one lane per run, at most n runs
    if (blocks > (int64_t)sm_count() * 16) blocks = (int64_t)sm_count() * 16;
    const int grid = (int)(blocks < 1 ? 1 : blocks);
#define HB_RES(MODE, PEER)                                                                              \
  HB_LAUNCH((runs_resolve_kernel<MODE, PEER>), grid, kBlock, 0, st, h->view, *runs, rs,                \
            (const char*)cache_rows, row_bytes, vb, f.run_src, slots, err)
    if (mode == HB_LOOKUP_SORTED) {
      if (table) HB_RES(HB_LOOKUP_SORTED, true); else HB_RES(HB_LOOKUP_SORTED, false);
    } else {
      if (table) HB_RES(HB_LOOKUP_SETASSOC, true); else HB_RES(HB_LOOKUP_SETASSOC, false);
    }
#undef HB_RES
  }
  if (resolve && sharded)
    HB_LAUNCH(runs_stage_kernel, sm_count() * 4, kBlock, 0, st, *runs, rs, row_bytes, vb);
  if (resolve && dv && dv->requests) {
    int rc = a2a_direct_publish(dv->requests, *dv->parity_out, f.req_counts, st);
    if (rc != HB_OK) return rc;
  }
  if (!expand) return HB_OK;  // per distinct id only: slots in run_slots, remote rows staged or asked for
  const int per = items_per_warp(runs->n);
  const int grid = grid_of_warps(runs->n, per, kBlock, 32);
  Maintain none;
  memset(&none, 0, sizeof(none));
  // (a call that only expands does not know what wrote the rows, nor whether it still runs)
#define HB_EXP_F(PEER, RB, FULL)                                                                              \
  HB_LAUNCH_NEXT_IF(resolve, (runs_expand_kernel<PEER, RB, false, FULL>), grid, kBlock, 0, st, *runs, f.run_src, slots, \
                    row_bytes, vb, (char*)out_rows, locs, found, per, none)
#define HB_EXP(PEER, RB)                                               \
  do {                                                                       \
    if (RB != 0 && per == 32) HB_EXP_F(PEER, RB, RB != 0); else HB_EXP_F(PEER, RB, false); \
  } while (0)
#define HB_EXP_V(PEER)                                \
  do {                                                \
    if (v16 && row_bytes == 512) HB_EXP(PEER, 512);   \
    else if (v16) HB_EXP(PEER, 16);                   \
    else HB_EXP(PEER, 0);                             \
  } while (0)
  if (sharded || (dv && dv->peer_sources)) HB_EXP_V(true); else HB_EXP_V(false);
#undef HB_EXP_V
#undef HB_EXP
#undef HB_EXP_F
  return HB_OK;
}
}  // namespace

}  // extern "C"

int hb::runs_expand_maintain(const hb_runs_t* runs, const unsigned long long* run_src, const int64_t* run_slots,
                             const void* cache_rows, const void* table, int64_t row_bytes, void* out_rows,
                             int64_t* locs, uint8_t* found, const Maintain& duty, cudaStream_t st) {
  const uintptr_t bits = (uintptr_t)row_bytes | (uintptr_t)cache_rows | (uintptr_t)out_rows | (uintptr_t)table;
  HB_CHECK_ARG((bits & 1) == 0, "hb_step_forward: rows must start at even addresses");
  const bool v16 = (bits & 15) == 0;
  const int vb = v16 ? 16 : ((bits & 3) == 0 ? 4 : 1);
  const int per = items_per_warp(runs->n);
  const int grid = grid_of_warps(runs->n, per, kBlock, 32) + duty.blocks;
#define HB_EXP_F(RB, FULL)                                                                                       \
  HB_LAUNCH_NEXT((runs_expand_kernel<false, RB, true, FULL>), grid, kBlock, 0, st, *runs, run_src, run_slots, row_bytes, \
            vb, (char*)out_rows, locs, found, per, duty)
#define HB_EXP(RB)                                         \
  do {                                                           \
    if (RB != 0 && per == 32) HB_EXP_F(RB, RB != 0); else HB_EXP_F(RB, false); \
  } while (0)
  if (v16 && row_bytes == 512) HB_EXP(512);
  else if (v16) HB_EXP(16);
  else HB_EXP(0);
#undef HB_EXP
#undef HB_EXP_F
  return HB_OK;
}

extern "C" {

size_t hb_lookup_fetch_runs_workspace_bytes(int64_t n, int64_t row_bytes, int sharded) {
  return make_fetch_plan(nullptr, n, row_bytes > 0 ? row_bytes : 1, sharded != 0).total;
}

int hb_lookup_fetch_runs(hb_index_t* h, const hb_runs_t* runs, const void* cache_rows,
                         const void* backing_rows, int64_t backing_num_rows, hb_peer_table_t* table,
                         int64_t row_bytes, void* out_rows, int64_t* locs, uint8_t* found,
                         int64_t* run_slots, int mode, void* workspace, size_t workspace_bytes,
                         hb_stream_t stream) {
  return fetch_runs_impl(h, runs, cache_rows, backing_rows, backing_num_rows, table, row_bytes, out_rows, locs,
                         found, run_slots, mode, workspace, workspace_bytes, stream, nullptr, true,
                         out_rows != nullptr);
}

int hb_runs_resolve_requests(hb_index_t* h, const hb_runs_t* runs, const void* cache_rows,
                             hb_peer_table_t* table, int64_t row_bytes, void* stage_rows, int64_t stage_cap,
                             int64_t* run_slots, hb_a2a_t* requests, int* parity_out, int mode, void* workspace,
                             size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(table && stage_rows && stage_cap > 0 && requests && parity_out,
               "hb_runs_resolve_requests: null argument");
  HB_CHECK_ARG(((uintptr_t)stage_rows & 15) == 0, "hb_runs_resolve_requests: the stage is 16-byte aligned");
  Delivery dv{(char*)stage_rows, stage_cap, requests, parity_out, true};
  return fetch_runs_impl(h, runs, cache_rows, nullptr, 0, table, row_bytes, nullptr, nullptr, nullptr, run_slots,
                         mode, workspace, workspace_bytes, stream, &dv, true, false);
}

int hb_runs_expand(const hb_runs_t* runs, const void* cache_rows, const void* other_rows, int64_t row_bytes,
                   int peer_sources, void* out_rows, int64_t* locs, uint8_t* found, const int64_t* run_slots,
                   void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(out_rows != nullptr && cache_rows != nullptr, "hb_runs_expand: null argument");
  Delivery dv{(char*)other_rows, 0, nullptr, nullptr, peer_sources != 0};
  return fetch_runs_impl(nullptr, runs, cache_rows, nullptr, 0, nullptr, row_bytes, out_rows, locs, found,
                         const_cast<int64_t*>(run_slots), HB_LOOKUP_SETASSOC, workspace, workspace_bytes, stream,
                         &dv, false, true);
}

size_t hb_runs_miss_list_workspace_bytes(int64_t n) { return compact_workspace_bytes(n); }

int hb_runs_miss_list(const hb_runs_t* runs, const int64_t* locs, int locs_kind, int want_class,
                      int64_t cap, int64_t* miss_ids, int64_t* miss_src, int64_t* miss_count,
                      void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(runs && locs && miss_ids && miss_src && miss_count && cap > 0,
               "hb_runs_miss_list: null argument");
  HB_CHECK_ARG(locs_kind >= 0 && locs_kind <= 2, "hb_runs_miss_list: locs_kind is 0, 1 or 2");
  HB_CHECK_ARG(want_class < 0 || runs->dclass || runs->n == 0,
               "hb_runs_miss_list: the runs were built without a class table");
  cudaStream_t st = (cudaStream_t)stream;
  // entries beyond the count hold -1, which the index's add() ignores
  int64_t blocks = ceil_div(cap, kBlock);
  if (blocks > (int64_t)sm_count() * 8) blocks = (int64_t)sm_count() * 8;
  HB_LAUNCH(fill_i64_kernel, (int)blocks, kBlock, 0, st, miss_ids, cap, (int64_t)-1);
  if (runs->n == 0) {
    HB_CUDA(cudaMemsetAsync(miss_count, 0, sizeof(int64_t), st));
    return HB_OK;
  }
  MissPolicy pol{*runs, locs, locs_kind, want_class, cap, miss_ids, miss_src, miss_count};
  return run_compact(pol, runs->n, workspace, workspace_bytes, st);
}

}  // extern "C"
