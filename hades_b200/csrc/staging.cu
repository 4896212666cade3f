// Cold-gradient staging table in HBM: accumulate, flush and insert.  Replaces the
// arithmetic of the reference's cache-server process (python/EmbCache/server.py:
// _accumulate_gradients_cold_remote/_local :546-574, _send_staled_gradients
// :346-497, _update_cache :499-544), which does it with torch CPU indexing on
// shared-memory tensors behind sockets.
#include "index.cuh"
#include <type_traits>

#include "partition_core.cuh"
#include "staging.cuh"

namespace hb {
namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ int64_t effective_n(int64_t n, const int64_t* n_dev) {
  if (!n_dev) return n;
  const int64_t d = *n_dev;
  return d < n ? d : n;
}

// rows[q] of the warp's 32 items: dst_row += src_row (fp32), 4 rows in flight
template <int VEC>
__device__ __forceinline__ void warp_add_rows(const float* src_row, float* dst_row, bool active,
                                              int64_t dim) {
  const int lane = threadIdx.x & 31;
  const unsigned act = __ballot_sync(0xffffffffu, active);
  if (act == 0u) return;
  const unsigned long long sb = (unsigned long long)src_row;
  const unsigned long long db = (unsigned long long)dst_row;
  for (int q0 = 0; q0 < 32; q0 += 4) {
    if (((act >> q0) & 0xfu) == 0u) continue;
    const float* s[4];
    float* d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned long long a = __shfl_sync(0xffffffffu, sb, q0 + u);
      const unsigned long long b = __shfl_sync(0xffffffffu, db, q0 + u);
      const bool on = (act >> (q0 + u)) & 1u;
      s[u] = on ? reinterpret_cast<const float*>(a) : nullptr;
      d[u] = reinterpret_cast<float*>(b);
    }
    if (VEC == 4) {
      const int64_t vpr = dim >> 2;
      for (int64_t k = lane; k < vpr; k += 32) {
        float4 x[4], y[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (s[u]) {
            x[u] = __ldcg(reinterpret_cast<const float4*>(s[u]) + k);
            y[u] = reinterpret_cast<float4*>(d[u])[k];
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (s[u]) {
            y[u].x += x[u].x; y[u].y += x[u].y; y[u].z += x[u].z; y[u].w += x[u].w;
            reinterpret_cast<float4*>(d[u])[k] = y[u];
          }
      }
    } else {
      for (int64_t k = lane; k < dim; k += 32) {
        float x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (s[u]) x[u] = s[u][k];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (s[u]) d[u][k] += x[u];
      }
    }
  }
}

// ---- accumulate through the cache index (cold remote, server.py:546-562) --------------
// Bound by row traffic (read, read, write of 512 bytes at random places).  Three blocks on an SM: 100,000
// rows, 391 blocks, took a wave and a third with the two that 112 registers allow (37.5 -> 31.0 us), and no
// store that waits for a load stands ahead of the rows (31.4 -> 28.4).  The sorted lookup keeps its top level in
// shared memory and stays at two.
template <int MODE, int VEC>
__global__ void __launch_bounds__(kBlock, MODE == HB_LOOKUP_SETASSOC ? 3 : 2) staging_accumulate_cached_kernel(
    IndexView v, hb_staging_t s, const int64_t* ids, const float* grads, int64_t n, const int64_t* n_dev,
    const int32_t* thr_table, int32_t default_thr, unsigned long long* dropped, int64_t* locs_out, int per) {
  begin_after_previous();
  __shared__ int64_t s_top[MODE == HB_LOOKUP_SORTED ? kTopMax : 1];
  if (MODE == HB_LOOKUP_SORTED) {
    stage_top_level(v, s_top);
    __syncthreads();
  }
  n = effective_n(n, n_dev);
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = warp * per; base < n; base += nwarps * per) {
    const int64_t i = lane < per ? base + lane : n;
    const int64_t id = i < n ? ids[i] : -1;
    const int64_t slot = warp_lookup<MODE>(v, s_top, id);
    const bool hit = slot >= 0;
    if (locs_out && i < n) locs_out[i] = slot;
    int32_t count = 0, limit = default_thr;  // (on their way with the rows)
    if (hit) {
      count = s.cnt[slot];
      if (thr_table) limit = thr_table[id];
    }
    warp_add_rows<VEC>(grads + i * s.dim, s.grad + (hit ? slot : 0) * s.dim, hit, s.dim);
    if (hit) {
      s.idx[slot] = id;
      s.iter_threshold[slot] = limit;
      s.cnt[slot] = count + 1;
    }
    if (dropped) {
      const unsigned miss = __ballot_sync(0xffffffffu, i < n && id >= 0 && !hit);
      if (lane == 0 && miss) atomicAdd(dropped, (unsigned long long)__popc(miss));
    }
  }
}

// ---- accumulate by direct address (cold local, server.py:564-574) -----------------------
template <int VEC>
__global__ void __launch_bounds__(kBlock) staging_accumulate_direct_kernel(
    hb_staging_t s, const int64_t* __restrict__ ids, const float* __restrict__ grads, int64_t n,
    const int64_t* __restrict__ n_dev, int64_t id_offset, int64_t id_stride) {
  n = effective_n(n, n_dev);
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t base = warp * 32; base < n; base += nwarps * 32) {
    const int64_t i = base + lane;
    const int64_t id = i < n ? __ldg(ids + i) : -1;
    int64_t slot = -1;
    if (id >= id_offset) {
      slot = (id - id_offset) / id_stride;
      if (slot >= s.slots) slot = -1;
    }
    const bool ok = slot >= 0;
    if (ok) {
      s.idx[slot] = id;
      s.cnt[slot] += 1;
    }
    warp_add_rows<VEC>(grads + i * s.dim, s.grad + (ok ? slot : 0) * s.dim, ok, s.dim);
  }
}

// ---- flush (server.py:346-425 remote / :427-497 local) ---------------------------------------
// Item = staging slot.  A slot is stale when cnt > 0 and (iter_count >=
// iter_threshold or cnt >= cnt_threshold); stale rows leave in slot order,
// bucketed by id % num_clients, and the slot is cleared; live slots with cnt > 0
// age by one iteration.
//
// One client: two launches.  flush_select_kernel reads the table's words once, ages the live slots and
// leaves one bit per stale slot and one count per block; flush_leave_kernel gives every block its place
// (the counts ahead of it), lists the stale slots of 1,024 in shared memory and takes them out, the rows as
// one run of vectors over the whole block, so that a block with a few per cent of its slots stale has all
// its threads on rows.  The selection waits for memory once per round of four words a warp; the second
// launch is bound by row traffic.  500,000 slots of 128 floats, 25,000 stale: 57 us in five launches
// (histogram, scan, scatter, move, a copy of the count), 54 without the copy -> 21.5.
struct FlushPlan {
  int64_t per_block;  // slots, a multiple of kFlushRound
  int blocks;
  uint32_t* masks;    // one bit per slot: stale
  int32_t* found;     // [blocks]
};
constexpr int kFlushRound = 1024;     // slots a block selects or lists at a time
constexpr int kFlushBlocksMax = 4096; // every block adds up the counts ahead of it

int64_t flush_rounds(int64_t slots) { return ceil_div(slots, (int64_t)kFlushRound); }
size_t flush_mask_bytes(int64_t slots) { return align_up((size_t)flush_rounds(slots) * (kFlushRound / 8), 256); }

FlushPlan flush_plan(void* ws, int64_t slots) {
  const int64_t rounds = flush_rounds(slots), per = ceil_div(rounds, (int64_t)kFlushBlocksMax);
  FlushPlan p;
  p.per_block = per * kFlushRound;
  p.blocks = (int)ceil_div(rounds, per);
  p.masks = static_cast<uint32_t*>(ws);
  p.found = reinterpret_cast<int32_t*>(static_cast<char*>(ws) + flush_mask_bytes(slots));
  return p;
}

__global__ void __launch_bounds__(kBlock) flush_select_kernel(hb_staging_t s, int32_t cnt_threshold, FlushPlan p) {
  begin_after_previous();
  __shared__ int s_found[kBlock / 32];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int64_t begin = blockIdx.x * p.per_block;
  const int64_t end = begin + p.per_block < s.slots ? begin + p.per_block : s.slots;
  int found = 0;
  for (int64_t base = begin; base < end; base += kFlushRound) {
    const int64_t first = base + warp * 128 + lane;
    int32_t c[4], age[4], limit[4];
    int64_t id[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = first + 32 * k < end ? s.cnt[first + 32 * k] : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      age[k] = limit[k] = 0;
      id[k] = -1;
      if (c[k] > 0) {
        age[k] = s.iter_count[first + 32 * k];
        limit[k] = s.iter_threshold[first + 32 * k];
        id[k] = s.idx[first + 32 * k];
      }
    }
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool stale = c[k] > 0 && (age[k] >= limit[k] || c[k] >= cnt_threshold) && id[k] >= 0;
      if (c[k] > 0 && !stale) s.iter_count[first + 32 * k] = age[k] + 1;  // server.py:418
      const uint32_t word = __ballot_sync(0xffffffffu, stale);
      if (lane == k) mine = word;
      found += __popc(word);
    }
    if (lane < 4) p.masks[(base >> 5) + warp * 4 + lane] = mine;
  }
  if (lane == 0) s_found[warp] = found;
  __syncthreads();
  if (threadIdx.x == 0) {
    int all = 0;
    for (int w = 0; w < kBlock / 32; ++w) all += s_found[w];
    p.found[blockIdx.x] = all;
  }
}

// VB: bytes per vector of a row
template <int VB>
__global__ void __launch_bounds__(kBlock) flush_leave_kernel(
    hb_staging_t s, FlushPlan p, int64_t out_cap, int64_t* line_ids, int32_t* lru, int64_t* out_ids, float* out_rows,
    int64_t* out_cnt, int64_t* counts, int64_t* host_count) {
  begin_after_previous();
  using V = typename std::conditional<VB == 16, uint4, uint32_t>::type;
  __shared__ int s_sum[kBlock / 32];
  __shared__ uint16_t s_list[kFlushRound];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int here = p.found[blockIdx.x];
  if (blockIdx.x > 0 && here == 0) return;
  // the counts ahead of this block; block 0 (its place is 0) adds up all of them
  const int upto = blockIdx.x > 0 ? (int)blockIdx.x : p.blocks;
  int sum = 0;
  for (int b = threadIdx.x; b < upto; b += kBlock) sum += p.found[b];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) s_sum[warp] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int w = 0; w < kBlock / 32; ++w) sum += s_sum[w];
  int64_t at = sum;
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) {
      counts[0] = sum;
      if (host_count) *reinterpret_cast<volatile int64_t*>(host_count) = sum;
    }
    if (here == 0) return;
    at = 0;
  }
  const int64_t vpr = (int64_t)s.dim * 4 / VB;
  const int64_t step_row = kBlock / vpr, step_vec = kBlock % vpr;
  V zero;
  memset(&zero, 0, sizeof(zero));
  const int64_t begin = blockIdx.x * p.per_block;
  const int64_t end = begin + p.per_block < s.slots ? begin + p.per_block : s.slots;
  for (int64_t base = begin; base < end; base += kFlushRound) {
    const uint32_t word = p.masks[(base >> 5) + lane];
    int ahead = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, ahead, o);
      if (lane >= o) ahead += t;
    }
    const int stale = __shfl_sync(0xffffffffu, ahead, 31);
    ahead -= __popc(word);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = __shfl_sync(0xffffffffu, word, warp * 4 + k);
      const int to = __shfl_sync(0xffffffffu, ahead, warp * 4 + k);
      if ((w >> lane) & 1u) s_list[to + __popc(w & ((1u << lane) - 1u))] = (uint16_t)((warp * 4 + k) * 32 + lane);
    }
    __syncthreads();
    const int64_t room = out_cap - at;
    const int leave = room <= 0 ? 0 : (room < stale ? (int)room : stale);
    for (int e = threadIdx.x; e < stale; e += kBlock) {
      const int64_t slot = base + s_list[e];
      if (e < leave) {
        const int64_t id = s.idx[slot];
        out_ids[at + e] = id;
        out_cnt[at + e] = (int64_t)s.cnt[slot];
        s.cnt[slot] = 0;  // server.py:419
        s.iter_count[slot] = 0;
        if (line_ids && line_ids[slot] == id) {  // _idx_cache.reset(ids), server.py:413
          line_ids[slot] = -1;
          lru[slot] = 0;
        }
      } else {
        s.iter_count[slot] += 1;  // the output has no room for it: it waits for the next flush
      }
    }
    int64_t row = threadIdx.x / vpr, k = threadIdx.x % vpr;
    while (row < leave) {
      V* src[4];
      V v[4];
      V* dst[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        src[u] = nullptr;
        if (row < leave) {
          src[u] = reinterpret_cast<V*>(s.grad + (base + s_list[row]) * s.dim) + k;
          dst[u] = reinterpret_cast<V*>(out_rows + (at + row) * s.dim) + k;
          v[u] = *src[u];
        }
        row += step_row;
        k += step_vec;
        if (k >= vpr) {
          k -= vpr;
          ++row;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (src[u]) {
          *dst[u] = v[u];
          *src[u] = zero;
        }
    }
    at += stale;
    __syncthreads();
  }
}

// Several clients: the partition selects: it writes the id of every stale slot to its place in
// the output (slot order within a bucket), leaves the slot number where the count will go,
// resets the cache entry and ages the live slots; no row moves there, because with a few
// per cent of the slots stale a warp of the partition would move one or two rows at a time.
// The second pass runs over the stale entries only: count out and cleared, row out and zeroed.
struct FlushPolicy {
  hb_staging_t s;
  int32_t cnt_threshold;
  int num_clients;
  int64_t* line_ids;  // nullable: the cache index entries of flushed ids are reset
  int32_t* lru;
  int64_t* out_ids;
  int64_t* out_cnt;   // holds the slot number until the second pass
  __device__ __forceinline__ int classify(int64_t i) const {
    const int32_t c = s.cnt[i];
    if (c <= 0) return -1;
    if (!(s.iter_count[i] >= s.iter_threshold[i] || c >= cnt_threshold)) return -1;
    const int64_t id = s.idx[i];
    return id >= 0 ? (int)mod_nonneg(id, num_clients) : -1;
  }
  __device__ __forceinline__ void emit(int64_t i, int, int64_t pos, int64_t start,
                                       bool active) const {
    const int64_t d = start + pos;
    if (active) {
      const int64_t id = s.idx[i];
      out_ids[d] = id;
      out_cnt[d] = i;
      if (line_ids && line_ids[i] == id) {  // _idx_cache.reset(ids), server.py:413
        line_ids[i] = -1;
        lru[i] = 0;
      }
    } else if (i < s.slots && s.cnt[i] > 0) {
      s.iter_count[i] += 1;  // server.py:418
    }
  }
};

// Second pass of the flush: entry d < sum(counts) left slot out_cnt[d]; its count goes out
// and starts again (server.py:419), its row goes out and is zeroed.  VB: bytes per vector.
template <int VB>
__global__ void __launch_bounds__(kBlock) staging_flush_move_kernel(
    hb_staging_t s, const int64_t* __restrict__ counts, int num_clients, int64_t out_cap,
    int64_t* __restrict__ out_cnt, float* __restrict__ out_rows) {
  using V = typename std::conditional<VB == 16, uint4, uint32_t>::type;
  int64_t total = 0;
  for (int c = 0; c < num_clients; ++c) total += counts[c];
  if (total > out_cap) total = out_cap;
  const int lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t vpr = (int64_t)s.dim * 4 / VB;
  V zero;
  memset(&zero, 0, sizeof(zero));
  for (int64_t base = warp * 32; base < total; base += nwarps * 32) {
    const int64_t d = base + lane;
    int64_t slot = -1;
    if (d < total) {
      slot = out_cnt[d];
      out_cnt[d] = (int64_t)s.cnt[slot];
      s.cnt[slot] = 0;
      s.iter_count[slot] = 0;
    }
    const int rows_here = (int)((total - base) < 32 ? (total - base) : 32);
    for (int q0 = 0; q0 < rows_here; q0 += 4) {
      V* src[4];
      V* dst[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int64_t sl = __shfl_sync(0xffffffffu, slot, (q0 + u) & 31);
        const bool on = q0 + u < rows_here;
        src[u] = on ? reinterpret_cast<V*>(s.grad + sl * s.dim) : nullptr;
        dst[u] = reinterpret_cast<V*>(out_rows + (base + q0 + u) * s.dim);
      }
      for (int64_t k = lane; k < vpr; k += 32) {
        V v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (src[u]) v[u] = src[u][k];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (src[u]) {
            __stcs(dst[u] + k, v[u]);
            src[u][k] = zero;
          }
      }
    }
  }
}

// ---- insert (server.py:499-544): rows into the cache buffer at the slots add() gave ----------
// Bound by row traffic: a row read, a cache row and a staging row written, all at random places.  Of a warp's 32
// entries a part has a row to move (of the distinct ids of a batch some 30 to 45 per cent); moved where they stand,
// four of 32 at a time, one or two rows of a warp were on their way together.  So the warp closes the gaps first.
// (512-byte rows, us: 700 of 2,000 entries 4.9 -> 3.0, 20,000 8.0 -> 6.2, 76,000 of 227,000 33.3 -> 28.9, 4.0 TB/s;
// 100,000 of 100,000 36.3 -> 33.2, 4.6 TB/s.)

// `rows` rows of vpr 16-byte vectors, lane r holds those of row r: copied (or zeroed where SRC is false)
template <bool SRC>
__device__ __forceinline__ void warp_put_rows(unsigned long long src, unsigned long long dst, int rows, int vpr) {
  constexpr int kFly = 8;
  const int lane = lane_id();
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  int glog2 = 5;
  while (glog2 > 0 && (1 << (glog2 - 1)) >= vpr) --glog2;
  const int rpp = 32 >> glog2, sub = lane & ((1 << glog2) - 1), which = lane >> glog2;
  for (int q0 = 0; q0 < rows; q0 += kFly * rpp) {
    for (int k0 = 0; k0 < vpr; k0 += 32) {
      const int k = k0 + sub;
      uint4 v[kFly];
      if (SRC) {
#pragma unroll
        for (int x = 0; x < kFly; ++x) {
          const int q = q0 + x * rpp + which;
          const unsigned long long from = __shfl_sync(0xffffffffu, src, q & 31);
          if (q < rows && k < vpr) v[x] = load_settled(reinterpret_cast<const uint4*>(from) + k);
        }
      }
#pragma unroll
      for (int x = 0; x < kFly; ++x) {
        const int q = q0 + x * rpp + which;
        const unsigned long long to = __shfl_sync(0xffffffffu, dst, q & 31);
        if (q < rows && k < vpr) reinterpret_cast<uint4*>(to)[k] = SRC ? v[x] : zero;
      }
    }
  }
}

// VEC_BYTES of a cached row; ZERO16: staging rows are zeroed in vectors of 16 bytes
template <int VEC_BYTES, bool ZERO16>
__global__ void __launch_bounds__(kBlock, 4) staging_insert_kernel(
    hb_staging_t s, const int64_t* locs, const uint8_t* last_writer, const char* emb_rows, const int64_t* row_index,
    char* cache_rows, int64_t row_bytes, int64_t n, const int64_t* n_dev) {
  begin_after_previous();
  __shared__ uint8_t s_at[kBlock / 32][32];
  n = effective_n(n, n_dev);
  const int lane = lane_id();
  uint8_t* const mine = s_at[threadIdx.x >> 5];
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  // Every warp has its share, of the warps that run at once (a round of 32 a warp: five warps' work on four warps' places
  // for 76,000 new ids among 175,000; a step of 65,536 ids 113.3 -> 111.7 us, others the same).
  const int64_t end = n * (warp + 1) / nwarps;
  for (int64_t base = n * warp / nwarps; base < end; base += 32) {
    const int64_t i = base + lane;
    const int64_t loc = i < end ? locs[i] : -1;
    const int64_t row = i < end && row_index ? row_index[i] : i;  // row of entry i in emb_rows
    // of several ids that received the same slot, the last of the batch writes it
    const bool ok = i < end && last_writer[i] && loc >= 0;
    const unsigned act = __ballot_sync(0xffffffffu, ok);
    if (act == 0u) continue;
    const int rows = __popc(act);
    if (ok) {
      if (s.cnt) {
        s.cnt[loc] = 0;   // server.py:539-541
        s.idx[loc] = -1;
      }
      mine[__popc(act & ((1u << lane) - 1u))] = (uint8_t)lane;
    }
    __syncwarp();
    const int at = lane < rows ? mine[lane] : 0;  // the lane whose row this one holds from here on
    __syncwarp();
    const int64_t slot = __shfl_sync(0xffffffffu, loc, at);
    const char* src = emb_rows + __shfl_sync(0xffffffffu, row, at) * row_bytes;
    char* dst = cache_rows + slot * row_bytes;
    if (VEC_BYTES == 16)
      warp_put_rows<true>((unsigned long long)src, (unsigned long long)dst, rows, (int)(row_bytes >> 4));
    else
      warp_move_rows(src, dst, lane < rows, row_bytes, VEC_BYTES);
    if (!s.grad) continue;
    if (ZERO16) {
      warp_put_rows<false>(0ull, (unsigned long long)(s.grad + slot * s.dim), rows, (int)(s.dim >> 2));
    } else {
      for (int q = 0; q < rows; ++q) {
        float* to = s.grad + __shfl_sync(0xffffffffu, slot, q) * s.dim;
        for (int64_t k = lane; k < s.dim; k += 32) to[k] = 0.f;
      }
    }
  }
}

int warp_grid(int64_t n) {
  int64_t blocks = ceil_div(ceil_div(n, 32) * 32, kBlock);
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

int check_staging(const hb_staging_t* s, const char* who) {
  if (!s || !s->grad || !s->cnt || !s->idx || !s->iter_count || !s->iter_threshold ||
      s->slots <= 0 || s->dim <= 0) {
    set_error("%s: incomplete staging table description", who);
    return HB_ERR_INVALID;
  }
  return HB_OK;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hb_staging_accumulate_cached(hb_index_t* h, const hb_staging_t* s, const int64_t* ids,
                                 const float* grads, int64_t n, const int64_t* n_dev,
                                 const int32_t* threshold_table, int32_t default_threshold,
                                 int mode, int64_t* dropped, int64_t* locs_out,
                                 hb_stream_t stream) {
  HB_CHECK_ARG(h != nullptr, "hb_staging_accumulate_cached: null index");
  int rc = check_staging(s, "hb_staging_accumulate_cached");
  if (rc) return rc;
  HB_CHECK_ARG(n >= 0 && (n == 0 || (ids && grads)), "hb_staging_accumulate_cached: null argument");
  HB_CHECK_ARG(s->slots == h->cache_size,
               "hb_staging_accumulate_cached: the staging table must have one slot per cache slot");
  HB_CHECK_ARG(mode == HB_LOOKUP_SETASSOC || mode == HB_LOOKUP_SORTED,
               "hb_staging_accumulate_cached: unknown mode");
  if (n == 0) return HB_OK;
  cudaStream_t st = (cudaStream_t)stream;
  if (mode == HB_LOOKUP_SORTED && h->sorted_stale) {
    rc = hb_index_build_sorted(h, stream);
    if (rc) return rc;
  }
  const bool vec4 = (s->dim % 4 == 0) && (((uintptr_t)grads | (uintptr_t)s->grad) & 15) == 0;
  const int per = items_per_warp(n);
  const int grid = grid_of_warps(n, per, kBlock, 16);
#define HB_ACC(MODE, VEC)                                                                     \
  HB_LAUNCH_NEXT((staging_accumulate_cached_kernel<MODE, VEC>), grid, kBlock, 0, st, h->view, *s,  \
            ids, grads, n, n_dev, threshold_table, default_threshold,                         \
            (unsigned long long*)dropped, locs_out, per)
  if (mode == HB_LOOKUP_SORTED) {
    if (vec4) HB_ACC(HB_LOOKUP_SORTED, 4); else HB_ACC(HB_LOOKUP_SORTED, 1);
  } else {
    if (vec4) HB_ACC(HB_LOOKUP_SETASSOC, 4); else HB_ACC(HB_LOOKUP_SETASSOC, 1);
  }
#undef HB_ACC
  return HB_OK;
}

int hb_staging_accumulate_direct(const hb_staging_t* s, const int64_t* ids, const float* grads,
                                 int64_t n, const int64_t* n_dev, int64_t id_offset,
                                 int64_t id_stride, hb_stream_t stream) {
  int rc = check_staging(s, "hb_staging_accumulate_direct");
  if (rc) return rc;
  HB_CHECK_ARG(n >= 0 && (n == 0 || (ids && grads)), "hb_staging_accumulate_direct: null argument");
  HB_CHECK_ARG(id_stride > 0, "hb_staging_accumulate_direct: id_stride must be positive");
  if (n == 0) return HB_OK;
  const bool vec4 = (s->dim % 4 == 0) && (((uintptr_t)grads | (uintptr_t)s->grad) & 15) == 0;
  if (vec4)
    HB_LAUNCH(staging_accumulate_direct_kernel<4>, warp_grid(n), kBlock, 0, (cudaStream_t)stream,
              *s, ids, grads, n, n_dev, id_offset, id_stride);
  else
    HB_LAUNCH(staging_accumulate_direct_kernel<1>, warp_grid(n), kBlock, 0, (cudaStream_t)stream,
              *s, ids, grads, n, n_dev, id_offset, id_stride);
  return HB_OK;
}

size_t hb_staging_flush_workspace_bytes(int64_t slots, int num_clients) {
  if (num_clients == 1) return flush_mask_bytes(slots > 0 ? slots : 1) + align_up(kFlushBlocksMax * sizeof(int32_t), 256);
  return partition_workspace_bytes(slots, num_clients);
}

int hb_staging_flush(hb_index_t* h, const hb_staging_t* s, int32_t cnt_threshold, int num_clients,
                     int64_t out_cap, int64_t* out_ids, float* out_rows, int64_t* out_cnt,
                     int64_t* counts, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  return hb_staging_flush_counted(h, s, cnt_threshold, num_clients, out_cap, out_ids, out_rows, out_cnt, counts, nullptr,
                                  workspace, workspace_bytes, stream);
}

int hb_staging_flush_counted(hb_index_t* h, const hb_staging_t* s, int32_t cnt_threshold, int num_clients,
                             int64_t out_cap, int64_t* out_ids, float* out_rows, int64_t* out_cnt, int64_t* counts,
                             int64_t* host_count, void* workspace, size_t workspace_bytes, hb_stream_t stream) {
  int rc = check_staging(s, "hb_staging_flush");
  if (rc) return rc;
  if (out_cap <= 0 || out_cap > s->slots) out_cap = s->slots;
  HB_CHECK_ARG(out_cap == s->slots || num_clients == 1,
               "hb_staging_flush: an output smaller than the table needs num_clients == 1");
  HB_CHECK_ARG(out_ids && out_rows && out_cnt && counts, "hb_staging_flush: null output");
  HB_CHECK_ARG(num_clients >= 1, "hb_staging_flush: num_clients must be positive");
  HB_CHECK_ARG(s->slots < ((int64_t)1 << 31), "hb_staging_flush: too many slots");
  HB_CHECK_ARG(!h || h->cache_size == s->slots,
               "hb_staging_flush: the staging table must have one slot per cache slot");
  HB_CHECK_ARG(!host_count || num_clients == 1, "hb_staging_flush: host_count needs num_clients == 1");
  const bool vec16 = payload_vec_bytes(s->dim * (int64_t)sizeof(float), s->grad, out_rows) == 16;
  if (num_clients == 1) {
    if (!workspace || workspace_bytes < hb_staging_flush_workspace_bytes(s->slots, 1)) {
      set_error("hb_staging_flush: workspace of %zu bytes needed, %zu given",
                hb_staging_flush_workspace_bytes(s->slots, 1), workspace_bytes);
      return HB_ERR_WORKSPACE;
    }
    const FlushPlan p = flush_plan(workspace, s->slots);
    int64_t* line_ids = h ? h->line_ids : nullptr;
    int32_t* lru = h ? h->lru : nullptr;
    HB_LAUNCH_NEXT(flush_select_kernel, p.blocks, kBlock, 0, (cudaStream_t)stream, *s, cnt_threshold, p);
    if (h) h->sorted_stale = true;
    if (vec16)
      HB_LAUNCH_NEXT(flush_leave_kernel<16>, p.blocks, kBlock, 0, (cudaStream_t)stream, *s, p, out_cap, line_ids, lru, out_ids,
                out_rows, out_cnt, counts, host_count);
    else
      HB_LAUNCH_NEXT(flush_leave_kernel<4>, p.blocks, kBlock, 0, (cudaStream_t)stream, *s, p, out_cap, line_ids, lru, out_ids,
                out_rows, out_cnt, counts, host_count);
    return HB_OK;
  }
  FlushPolicy pol{*s, cnt_threshold, num_clients, h ? h->line_ids : nullptr,
                  h ? h->lru : nullptr, out_ids, out_cnt};
  rc = run_partition(pol, s->slots, num_clients, workspace, workspace_bytes, counts,
                     (cudaStream_t)stream, 8);
  if (rc != HB_OK) return rc;
  if (h) h->sorted_stale = true;
  // the number of stale rows is only known on the device: size the grid for a full output
  const int grid = warp_grid(out_cap);
  if (vec16)
    HB_LAUNCH(staging_flush_move_kernel<16>, grid, kBlock, 0, (cudaStream_t)stream, *s, counts, num_clients,
              out_cap, out_cnt, out_rows);
  else
    HB_LAUNCH(staging_flush_move_kernel<4>, grid, kBlock, 0, (cudaStream_t)stream, *s, counts, num_clients,
              out_cap, out_cnt, out_rows);
  return HB_OK;
}

size_t hb_staging_insert_workspace_bytes(int64_t n) {
  return hb_index_add_workspace_bytes(n) + align_up((size_t)(n > 0 ? n : 1), 256);
}

int hb_staging_insert(hb_index_t* h, const hb_staging_t* s, const int64_t* ids,
                      const void* emb_rows, int64_t n, void* cache_rows, int64_t row_bytes,
                      int64_t* locs_out, void* workspace, size_t workspace_bytes,
                      hb_stream_t stream) {
  return hb_staging_insert_gather(h, s, ids, emb_rows, nullptr, n, cache_rows, row_bytes, locs_out,
                                  workspace, workspace_bytes, stream);
}

int hb_staging_insert_gather(hb_index_t* h, const hb_staging_t* s, const int64_t* ids,
                             const void* emb_rows, const int64_t* row_index, int64_t n,
                             void* cache_rows, int64_t row_bytes, int64_t* locs_out, void* workspace,
                             size_t workspace_bytes, hb_stream_t stream) {
  HB_CHECK_ARG(h != nullptr, "hb_staging_insert: null index");
  HB_CHECK_ARG(n >= 0 && row_bytes > 0, "hb_staging_insert: bad sizes");
  HB_CHECK_ARG(n == 0 || (ids && emb_rows && cache_rows && locs_out), "hb_staging_insert: null argument");
  HB_CHECK_ARG(!s || s->slots == h->cache_size,
               "hb_staging_insert: the staging table must have one slot per cache slot");
  if (n == 0) return HB_OK;
  const size_t flag_bytes = align_up((size_t)n, 256);
  if (!workspace || workspace_bytes < hb_staging_insert_workspace_bytes(n)) {
    set_error("hb_staging_insert: workspace of %zu bytes needed, %zu given",
              hb_staging_insert_workspace_bytes(n), workspace_bytes);
    return HB_ERR_WORKSPACE;
  }
  uint8_t* last_writer = static_cast<uint8_t*>(workspace);
  int rc = hb_index_add(h, ids, n, locs_out, last_writer, static_cast<char*>(workspace) + flag_bytes,
                        workspace_bytes - flag_bytes, stream);
  if (rc) return rc;
  return staging_insert_rows(s, emb_rows, row_index, n, nullptr, cache_rows, row_bytes, locs_out, last_writer, true,
                             (cudaStream_t)stream);
}

int hb_staging_insert_rows(const hb_staging_t* s, const void* emb_rows, const int64_t* row_index, int64_t n,
                           void* cache_rows, int64_t row_bytes, const int64_t* locs, const uint8_t* last_writer,
                           hb_stream_t stream) {
  return staging_insert_rows(s, emb_rows, row_index, n, nullptr, cache_rows, row_bytes, locs, last_writer, false,
                             (cudaStream_t)stream);
}

}  // extern "C"

int hb::staging_insert_rows(const hb_staging_t* s, const void* emb_rows, const int64_t* row_index, int64_t n,
                            const int64_t* n_dev, void* cache_rows, int64_t row_bytes, const int64_t* locs,
                            const uint8_t* last_writer, bool early, cudaStream_t st) {
  HB_CHECK_ARG(n >= 0 && row_bytes > 0, "hb_staging_insert_rows: bad sizes");
  HB_CHECK_ARG(n == 0 || (emb_rows && cache_rows && locs && last_writer), "hb_staging_insert_rows: null argument");
  if (n == 0) return HB_OK;
  hb_staging_t none;
  memset(&none, 0, sizeof(none));
  const hb_staging_t st_desc = s ? *s : none;
  const int vb = payload_vec_bytes(row_bytes, emb_rows, cache_rows);
  const bool zero16 = st_desc.dim % 4 == 0 && ((uintptr_t)st_desc.grad & 15) == 0;
#define HB_INSERT(VB, Z16)                                                                                     \
  HB_LAUNCH_NEXT_IF(early, (staging_insert_kernel<VB, Z16>), grid_of_warps(n, 4, kBlock, 4), kBlock, 0, st, st_desc, \
                    locs, last_writer, (const char*)emb_rows, row_index, (char*)cache_rows, row_bytes, n, n_dev)
  if (vb == 16) {
    if (zero16) HB_INSERT(16, true); else HB_INSERT(16, false);
  } else if (vb == 4) {
    if (zero16) HB_INSERT(4, true); else HB_INSERT(4, false);
  } else {
    if (zero16) HB_INSERT(1, true); else HB_INSERT(1, false);
  }
#undef HB_INSERT
  return HB_OK;
}
