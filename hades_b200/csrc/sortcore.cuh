// Stable sort of (key, position) pairs, fused with whatever works on the sorted order.
//
// A source says how many entries there are (a number that may only be known on the device) and
// what the key of entry i is; a finish takes the sorted chunk of every CTA and does the rest (run
// heads and classes of a batch, the walk over the cache sets, the LRU ageing) without another
// launch.  Least significant digit first, every pass
//   rank      warp by warp with match_any: how many earlier entries of the warp, of the CTA and of
//             the earlier CTAs have the same digit
//   scatter   to base[digit] + rank
// so that equal keys keep the order of the input.
//
// (kSkips: a source that usually has nothing to sort; the launch then ends at once and writes nothing.)
//
// What bounds it: latency.  A batch of 65,536 ids is half a megabyte, one of 2,000,000 is 16 MB and
// stays in L2; with one launch per pass the time goes into launches, cold starts and the chain of
// look-backs.  So
//  * the passes of one sort run in ONE launch, separated by barriers;
//  * digits are as wide as 10 bits and as few as the largest key needs, found on the device from
//    the OR of the keys (ids of a table of 20 M rows: 25 bits, three passes; a caller that says
//    nothing about its ids would pay eight passes of 8 bits otherwise);
//  * up to 65,536 entries a cluster of 1 to 16 CTAs does it all in (distributed) shared memory:
//    its barrier costs well under a microsecond and its digit counts are read from the peers' shared
//    memory directly;
//  * above that a cooperative grid, one CTA per SM, keeps its keys and ranks in registers between
//    the counting and the scatter of a pass and goes through L2; barriers are counters in the
//    workspace with bounded waits (gridbar.cuh).  A launch whose barrier runs out leaves an empty result
//    (give_up of its finish) for the launches behind it.
#pragma once

#include <cooperative_groups.h>

#include "gridbar.cuh"
#include "launch.cuh"

namespace hb {
int* device_error_word();  // runtime.cu

constexpr int kClusterT = 512;         // threads per CTA of the cluster version
constexpr int kClusterDigit = 8;       // its bits per pass: counts are exchanged between all CTAs
constexpr int kClusterMaxItems = 8;
constexpr int64_t kSortOneEach = 16 * (int64_t)kClusterT;  // ... with one entry per thread
// The cluster's largest input, and its line: it is ahead of the grid as far as its shared memory reaches (us,
// cluster / grid, ids of 21 bits: 24,000 21.4 / 30.8, 32,000 22.4 / 30.6, 45,000 28.2 / 31.5, 65,536 29.5 / 32.4).
constexpr int64_t kSortClusterMax = 16 * (int64_t)kClusterT * kClusterMaxItems;
static_assert(kSortClusterMax == kSortClusterEntries, "the line that launches behind a sort go by");
constexpr int kGridT = 1024;           // threads per CTA of the grid version
constexpr int kGridDigit = 10;
constexpr int kGridBins = 1 << kGridDigit;

// scratch of the grid version
struct SortGridBufs {
  uint2* kv0;          // [n]
  uint2* kv1;          // [n]
  uint32_t* hist;      // [grid][bins]
  unsigned* partial;   // [grid][4] OR of the keys (low, high), sentinel seen
  int4* exchange;      // [grid]
  unsigned* barrier;   // [kSortBarrierWords], zero before the launch, and with it the totals of the first pass
  uint32_t* groups;    // [2][kSortGroups][bins] counts of a group of CTAs; a pass and the next take turns
};
constexpr int kSortBarrierWords = 64;
// Groups of CTAs whose digit counts are added up by atomics: what lies ahead of a CTA is then the totals of the groups
// before its own and the counts of at most a dozen CTAs, read behind one barrier.  Offsets by columns that the CTAs scan
// among them cost a pass one barrier more, and adding up the counts of all CTAs ahead reads 44 MB a pass.  Together with
// barriers that arrive without waiting for the word (1.8 us before): 70,000 ids 45.4 -> 33.6 us, 282,624 49.4 -> 38.6,
// 524,288 59.2 -> 46.6, 1,048,576 78.7 -> 65.1, 2,000,000 119.5 -> 109.8.
constexpr int kSortGroups = 13;
__host__ __device__ inline int sort_group_ctas(int ctas) { return (ctas + kSortGroups - 1) / kSortGroups; }
static inline size_t sort_zero_words(int digit) { return kSortBarrierWords + ((size_t)kSortGroups << digit); }

static inline int sort_grid_ctas(int64_t n) {
  // Fewer CTAs where the chunks would get short: a barrier over few CTAs is quicker, and a CTA takes all registers of its SM,
  // so that what runs on other streams meanwhile needs an SM without one.  Up to 128 CTAs of 1,024 entries, which are two a
  // thread for half of its warps (70,000 ids 32.8 us, in half the CTAs 33.7), then of 2,048.  (A batch of add() with thousands
  // of copies of some ids, whose sets a thread walks at the end, is 1 to 4 % behind: 80,000 ids 4.57 -> 4.74 ms; of distinct
  // ids to few sets ahead: 80,000 to 20,000 places 95.9 -> 68.6 us, 100,000 to 50,000 102.7, with 2,048 for these lists 124.4.)
  int64_t g = ceil_div(n, n <= 128 * (int64_t)kGridT ? kGridT : 2 * kGridT);
  const int64_t cap = sm_count();
  return (int)(g > cap ? cap : (g < 1 ? 1 : g));
}

static inline size_t sort_grid_bytes(int64_t n) {
  if (n <= kSortClusterMax) return 0;
  const size_t g = (size_t)sm_count();
  return 2 * align_up((size_t)n * sizeof(uint2), 256) + align_up(g * kGridBins * 4, 256) + align_up(g * 16, 256) +
         align_up(g * sizeof(int4), 256) + kSortBarrierWords * 4 + (size_t)2 * kSortGroups * kGridBins * 4 + 256;
}

static inline SortGridBufs sort_grid_bufs(void* ws, int64_t n) {
  SortGridBufs b;
  Carver cv(ws);
  const size_t g = (size_t)sm_count();
  b.kv0 = cv.take<uint2>(n);
  b.kv1 = cv.take<uint2>(n);
  b.hist = cv.take<uint32_t>(g * kGridBins);
  b.partial = cv.take<unsigned>(g * 4);
  b.exchange = cv.take<int4>(g);
  b.barrier = cv.take<unsigned>(kSortBarrierWords + 2 * kSortGroups * kGridBins);
  b.groups = b.barrier + kSortBarrierWords;
  return b;
}

#ifdef __CUDACC__

namespace cg = cooperative_groups;

// key of an entry that takes no part: larger than any other at every width (all ones)
constexpr uint32_t kSortNone = 0xffffffffu;

// A source's entry i: fetch() brings its id, false where it takes no part; accept() makes the key of an id, false for
// one that is left out.  (Apart, so that the ids of a thread are on their way at once: what accept() does
// with a bad id kept the next load behind it.)
template <class Src>
__device__ __forceinline__ bool sort_load(const Src& src, int64_t i, unsigned long long& key) {
  int64_t id;
  return src.fetch(i, id) && src.accept(id, key);
}

struct SortDigits {
  int passes, width, bits;
  bool wide;  // keys of more than 32 bits: digits come from the source, by position
};

__device__ __forceinline__ SortDigits sort_digits(unsigned lo, unsigned hi, bool none_seen, int max_width) {
  SortDigits d;
  int bits = hi ? 64 - __clz(hi) : 32 - __clz(lo);
  if (none_seen) bits += 1;  // the all-ones key stays above every other
  if (bits < 1) bits = 1;
  if (bits > 64) bits = 64;
  d.wide = bits > 32;
  d.bits = bits;
  d.passes = (bits + max_width - 1) / max_width;
  d.width = (bits + d.passes - 1) / d.passes;
  return d;
}

// Digits from what the caller says of its keys (valid ones below 2^bits - 1), where that is as good as
// looking: not when one bit less would save a pass.  Spares an exchange between all CTAs.
__host__ __device__ inline bool sort_known_digits(int bits, int max_width, SortDigits& d) {
  if (bits <= 1 || bits > 30 || (bits + max_width - 1) / max_width != (bits - 1 + max_width - 1) / max_width) return false;
  d.wide = false;
  d.bits = bits;
  d.passes = (bits + max_width - 1) / max_width;
  d.width = (bits + d.passes - 1) / d.passes;
  return true;
}

// exclusive scan over the first `bins` threads of the CTA (bins <= 1024, a multiple of 32 or below
// 32); s_warp: [32].  All threads call it.
__device__ __forceinline__ uint32_t sort_block_exscan(uint32_t v, int bins, uint32_t* s_warp) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool on = warp * 32 < bins;
  uint32_t inc = v;
  if (on) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
  }
  __syncthreads();
  uint32_t before = 0;
  if (on) before = __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u);
  return before + inc - v;
}

// sums over the CTA's warps: `mine` is the same in every lane of a warp; before = the warps ahead.
// s4: [2 * W + 1].  A lane of four warps scans one component (a shuffle tree in every warp would
// take the CTA's shuffle unit a thousand cycles).
template <int W>
__device__ __forceinline__ void sort_warp_sums(const int4& mine, int4* s4, int4& before, int4& all) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s4[warp] = mine;
  __syncthreads();
  if (warp < 4) {
    const int v = lane < W ? reinterpret_cast<const int*>(s4 + lane)[warp] : 0;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane < W) reinterpret_cast<int*>(s4 + W + lane)[warp] = inc - v;
    if (lane == 31) reinterpret_cast<int*>(s4 + 2 * W)[warp] = inc;
  }
  __syncthreads();
  before = s4[W + warp];
  all = s4[2 * W];
}

// zero_masks: the words of sort_rank_warp too (they stay zero from then on)
template <int T>
__device__ __forceinline__ void sort_zero_counts(uint16_t* wcnt, uint32_t* wmask, int bins, int zero_masks) {
  uint32_t* w32 = reinterpret_cast<uint32_t*>(wcnt);
  const int words = (T / 32) * bins / 2;
  for (int k = threadIdx.x; k < words; k += T) w32[k] = 0u;
  for (int k = threadIdx.x; k < zero_masks; k += T) wmask[k] = 0u;
}

// rank of a warp's items among the earlier ones of the same digit in the warp; leaves the warp's
// digit counts in wc[0..bins).  wm[0..bins): one word per digit, zero before and after.
// The lanes that share a digit find each other through an atomic OR into wm: measured at 32 warps
// per SM 14 cycles per 32 items whose digits are scattered, against 60 for match.any (a turn for
// every distinct value) and 2.8 per vote for digit bits taken one by one.  Same-address atomics
// take turns, so neighbours that agree (popular ids once the lower digits are sorted) send one
// OR together.
template <int I>
__device__ __forceinline__ void sort_rank_warp(const uint32_t (&k)[I], int left, int shift,
                                               int width, uint16_t* wc, uint32_t* wm,
                                               uint32_t (&rank)[(I + 1) / 2]) {
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const uint32_t mask = (1u << width) - 1u;
  if (left + lane <= 0) return;  // the whole warp
#pragma unroll
  for (int i = 0; i < I; ++i) {
    const bool valid = i * 32 < left;
    const uint32_t d = valid ? (k[i] >> shift) & mask : ~0u;
    const uint32_t up = __shfl_up_sync(0xffffffffu, d, 1);
    const bool lead = lane == 0 || up != d;
    const unsigned leads = __ballot_sync(0xffffffffu, lead);
    if (lead && valid) {
      const unsigned later = leads & ~(lt | (1u << lane));
      const unsigned upto = later ? (later & (0u - later)) - 1u : ~0u;
      atomicOr(wm + d, upto & ~lt);
    }
    __syncwarp();
    uint32_t pre = 0, same = 0;
    if (valid) {
      pre = wc[d];
      same = wm[d];
    }
    __syncwarp();
    if (valid && (same & lt) == 0u) {
      wc[d] = (uint16_t)(pre + __popc(same));
      wm[d] = 0u;
    }
    __syncwarp();
    const uint32_t r = pre + __popc(same & lt);
    if (i & 1) rank[i >> 1] |= r << 16; else rank[i >> 1] = r;
  }
}

// counts per warp -> offsets of the warps inside the CTA, two digits per thread in one word (a
// CTA holds fewer than 65,536 entries); the CTA's counts go to total[0..bins)
template <int T>
__device__ __forceinline__ void sort_scan_warps(uint16_t* wcnt, int bins, uint32_t* total) {
  constexpr int W = T / 32;
  uint32_t* w32 = reinterpret_cast<uint32_t*>(wcnt);
  const int words = bins >> 1;
  for (int d = threadIdx.x; d < words; d += T) {
    uint32_t run = 0;
#pragma unroll
    for (int w0 = 0; w0 < W; w0 += 8) {
      uint32_t c[8];
#pragma unroll
      for (int w = 0; w < 8; ++w) c[w] = w32[(w0 + w) * words + d];
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        w32[(w0 + w) * words + d] = run;
        run += c[w];
      }
    }
    total[2 * d] = run & 0xffffu;
    total[2 * d + 1] = run >> 16;
  }
}

// ------------------------------------------------------------------------------------------------
// Cluster version: I entries per thread, chunk kClusterT * I per CTA, 1 to 16 CTAs of one cluster.
// ------------------------------------------------------------------------------------------------
struct SortClusterSmem {
  uint2* kv;         // [kClusterT * I]
  uint16_t* wcnt;    // [warps][bins]
  uint32_t* wmask;   // [warps][bins]
  uint32_t* total;   // [bins] read by the peers
  uint32_t* base;    // [bins]
  uint32_t* warp;    // [32]
  int4* sums;        // [2 * warps + 1]
  int4* cta4;        // [16 + 2]: stored by the peers; what lies ahead, all
  uint4* seen;       // [16]: stored by the peers
};

static inline size_t sort_cluster_smem_bytes(int items) {
  constexpr int W = kClusterT / 32, B = 1 << kClusterDigit;
  return (size_t)kClusterT * items * sizeof(uint2) + (size_t)W * B * 6 + 2 * B * 4 + 32 * 4 + (2 * W + 1) * sizeof(int4) +
         18 * sizeof(int4) + 16 * sizeof(uint4);
}

// what a finish sees: the sorted entries chunk by chunk, barriers and exchanges between the CTAs
template <int ITEMS>
struct ClusterCtx {
  static constexpr int kThreads = kClusterT;
  static constexpr int kItems = ITEMS;
  static constexpr int kChunk = kClusterT * ITEMS;
  static constexpr bool kBehindAll = false;
  // Stores of a finish behind its barrier, which would wait for them; its entries are kept in registers till then (the
  // grid has none to spare: 1,048,576 ids 62.5 -> 63.2 us, 2,000,000 103.6 -> 105.6).
  static constexpr bool kStoresLate = true;
  static_assert(ITEMS <= 8, "a chunk is a strip of eight entries a thread");
  SortClusterSmem s;
  int count;   // entries that were sorted
  uint32_t* scratch;  // shared memory, 8 * kThreads words, free after the sort
  int rank, ctas;
  bool wide;       // keys of more than 32 bits: .x of the entries is undefined
  bool none;       // some entries take no part (kSortNone)
  // (positions are 32-bit: at most 2^31 entries)
  // first entry of this lane (a warp takes 32 * kItems consecutive ones); item i is at + 32 * i
  __device__ __forceinline__ int first() const {
    return rank * kChunk + (threadIdx.x >> 5) * (32 * ITEMS) + (threadIdx.x & 31);
  }
  __device__ __forceinline__ uint32_t chunk_begin() const { return SortChunks(count, kChunk).begin(rank); }
  __device__ __forceinline__ uint32_t chunk_end() const { return SortChunks(count, kChunk).end(rank); }
  // a sorted entry of this chunk, or the last one of the chunk before: that one ahead of prefix() only (nobody's
  // shared memory is read after it, so that CTAs leave without waiting for each other)
  __device__ __forceinline__ uint2 get(int j) const {
    const int at = j - rank * kChunk;
    if (at >= 0) return s.kv[at];
    return *cg::this_cluster().map_shared_rank(s.kv + (kChunk + at), rank - 1);
  }
  // 8 consecutive ones of this chunk from a multiple of 8 on (those at and beyond `count` are undefined)
  __device__ __forceinline__ void get8(int j, uint2 (&e)[8]) const {
    const uint4* p = reinterpret_cast<const uint4*>(s.kv + (j - rank * kChunk));
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 x = p[q];
      e[2 * q] = make_uint2(x.x, x.y);
      e[2 * q + 1] = make_uint2(x.z, x.w);
    }
  }
  // sums over the CTAs: `mine` of the CTAs ahead and of all
  __device__ __forceinline__ bool prefix(const int4& mine, int4& before, int4& all) {
    if (ctas == 1) {
      before = make_int4(0, 0, 0, 0);
      all = mine;
      return true;
    }
    // stored at every peer: behind the barrier nobody waits for somebody else's shared memory
    if ((int)threadIdx.x < ctas) *cg::this_cluster().map_shared_rank(s.cta4 + rank, threadIdx.x) = mine;
    sync();
    if (threadIdx.x < 128) {  // a warp per component
      const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
      const int v = lane < ctas ? reinterpret_cast<const int*>(s.cta4 + lane)[c] : 0;
      const int b = __reduce_add_sync(0xffffffffu, lane < rank ? v : 0);
      const int a = __reduce_add_sync(0xffffffffu, v);
      if (lane == 0) {
        reinterpret_cast<int*>(s.cta4 + 16)[c] = b;
        reinterpret_cast<int*>(s.cta4 + 17)[c] = a;
      }
    }
    __syncthreads();
    before = s.cta4[16];
    all = s.cta4[17];
    return true;
  }
  // shared memory written before it, the peers' too, is seen after it
  __device__ __forceinline__ void sync() const {
    if (ctas > 1) cg::this_cluster().sync(); else __syncthreads();
  }
  // the same for global memory (read with __ldcg after it)
  __device__ __forceinline__ bool barrier() {
    if (ctas > 1) __threadfence();
    sync();
    return true;
  }
  // the sorted entries of all CTAs, read with __ldcg; buf: [count] in global memory
  __device__ __forceinline__ const uint2* publish(uint2* buf) {
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int j = first() + i * 32;
      if (j < count) __stcg(buf + j, s.kv[j - rank * kChunk]);
    }
    barrier();
    return buf;
  }
};

template <class Src, class Fin, int I>
__global__ void __launch_bounds__(kClusterT, 1) sort_cluster_kernel(Src src, Fin fin) {
  wait_for_previous();
  constexpr int T = kClusterT, W = T / 32, B = 1 << kClusterDigit;
  extern __shared__ __align__(16) char smem[];
  ClusterCtx<I> ctx;
  SortClusterSmem& s = ctx.s;
  {
    char* p = smem;
    s.kv = reinterpret_cast<uint2*>(p); p += (size_t)T * I * sizeof(uint2);
    s.wcnt = reinterpret_cast<uint16_t*>(p); p += (size_t)W * B * 2;
    s.wmask = reinterpret_cast<uint32_t*>(p); p += (size_t)W * B * 4;
    s.total = reinterpret_cast<uint32_t*>(p); p += B * 4;
    s.base = reinterpret_cast<uint32_t*>(p); p += B * 4;
    s.warp = reinterpret_cast<uint32_t*>(p); p += 32 * 4;
    s.sums = reinterpret_cast<int4*>(p); p += (2 * W + 1) * sizeof(int4);
    s.cta4 = reinterpret_cast<int4*>(p); p += 18 * sizeof(int4);
    s.seen = reinterpret_cast<uint4*>(p);
  }
  auto cluster = cg::this_cluster();
  ctx.scratch = s.wmask;
  ctx.rank = (int)cluster.block_rank();
  ctx.ctas = (int)cluster.num_blocks();
  const int n = (int)src.count();
  if (Src::kSkips && n == 0) return;
  ctx.count = n;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int first = ctx.first();
  uint32_t k[I], v[I];
  SortDigits dig;
  {
    unsigned lo = 0, hi = 0, none = 0;
    const bool known = sort_known_digits(src.known_bits(), kClusterDigit, dig);
    // (the peers have to run before something is stored at them)
    if (!known && ctx.ctas > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    int64_t id[I];
    unsigned part = 0u;
#pragma unroll
    for (int i = 0; i < I; ++i)
      if (first + i * 32 < n && src.fetch(first + i * 32, id[i])) part |= 1u << i;
#pragma unroll
    for (int i = 0; i < I; ++i) {
      const int j = first + i * 32;
      k[i] = kSortNone;
      v[i] = (uint32_t)j;
      if (j < n) {
        unsigned long long key;
        if (((part >> i) & 1u) && src.accept(id[i], key)) {
          k[i] = (uint32_t)key;
          lo |= (unsigned)key;
          hi |= (unsigned)(key >> 32);
        } else {
          none = 1u;
        }
      }
    }
    ctx.wide = false;
    ctx.none = true;
    if (!known) {
      lo = __reduce_or_sync(0xffffffffu, lo);
      hi = __reduce_or_sync(0xffffffffu, hi);
      none = __reduce_or_sync(0xffffffffu, none);
      uint4* per_warp = reinterpret_cast<uint4*>(s.sums);
      if (lane == 0) per_warp[warp] = make_uint4(lo, hi, none, 0u);
      __syncthreads();
      uint4 x = lane < W ? per_warp[lane] : make_uint4(0u, 0u, 0u, 0u);
      if (ctx.ctas > 1) {
        if (warp == 0) {
          x.x = __reduce_or_sync(0xffffffffu, x.x);
          x.y = __reduce_or_sync(0xffffffffu, x.y);
          x.z = __reduce_or_sync(0xffffffffu, x.z);
        }
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if ((int)threadIdx.x < ctx.ctas) *cluster.map_shared_rank(s.seen + ctx.rank, threadIdx.x) = x;
        ctx.sync();
        x = lane < ctx.ctas ? s.seen[lane] : make_uint4(0u, 0u, 0u, 0u);
      }
      x.x = __reduce_or_sync(0xffffffffu, x.x);
      x.y = __reduce_or_sync(0xffffffffu, x.y);
      x.z = __reduce_or_sync(0xffffffffu, x.z);
      dig = sort_digits(x.x, x.y, x.z != 0u, kClusterDigit);
      ctx.wide = dig.wide;
      ctx.none = x.z != 0u;
    }
  }
  for (int pass = 0; pass < dig.passes; ++pass) {
    const int bit = pass * dig.width;
    const int width = dig.bits - bit < dig.width ? dig.bits - bit : dig.width;
    const int bins = 1 << width;
    sort_zero_counts<T>(s.wcnt, s.wmask, bins, pass == 0 ? W * bins : 0);
    if (pass > 0) {
#pragma unroll
      for (int i = 0; i < I; ++i) {
        if (first + i * 32 < n) {
          const uint2 e = s.kv[warp * (32 * I) + i * 32 + lane];
          k[i] = e.x;
          v[i] = e.y;
        }
      }
    }
    if (dig.wide) {
#pragma unroll
      for (int i = 0; i < I; ++i)
        if (first + i * 32 < n) {
          unsigned long long key;
          k[i] = sort_load(src, v[i], key) ? (uint32_t)(key >> bit) : kSortNone;
        }
    }
    const int shift = dig.wide ? 0 : bit;
    __syncthreads();
    uint32_t rank[(I + 1) / 2];
    uint16_t* wc = s.wcnt + warp * bins;
    sort_rank_warp<I>(k, n - first, shift, width, wc, s.wmask + warp * bins, rank);
    __syncthreads();
    sort_scan_warps<T>(s.wcnt, bins, s.total);
    ctx.sync();
    uint32_t pre = 0, all = 0;
    if ((int)threadIdx.x < bins) {
      if (ctx.ctas > 1) {
        uint32_t t[16];  // all sixteen on their way at once
#pragma unroll
        for (int c = 0; c < 16; ++c) t[c] = c < ctx.ctas ? *cluster.map_shared_rank(s.total + threadIdx.x, c) : 0u;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          if (c < ctx.rank) pre += t[c];
          all += t[c];
        }
      } else {
        all = s.total[threadIdx.x];
      }
    }
    const uint32_t start = sort_block_exscan(all, bins, s.warp);
    if ((int)threadIdx.x < bins) s.base[threadIdx.x] = start + pre;
    __syncthreads();
    const uint32_t mask = bins - 1;
#pragma unroll
    for (int i = 0; i < I; ++i) {
      if (first + i * 32 < n) {
        const uint32_t d = (k[i] >> shift) & mask;
        const uint32_t to = s.base[d] + wc[d] + ((rank[i >> 1] >> (16 * (i & 1))) & 0xffffu);
        uint2* at = s.kv + (to & (T * I - 1));
        if (ctx.ctas > 1) at = cluster.map_shared_rank(at, to / (T * I));
        *at = make_uint2(k[i], v[i]);
      }
    }
    ctx.sync();
  }
  start_next();  // (from here on its start is hidden as well)
  fin.run(ctx, src);
}

// ------------------------------------------------------------------------------------------------
// Grid version: a cooperative launch, chunk of the input per CTA, scratch in global memory.
// ------------------------------------------------------------------------------------------------
template <int ITEMS>
struct GridCtx {
  static constexpr int kThreads = kGridT;
  static constexpr int kItems = ITEMS;
  static constexpr bool kStoresLate = false;
  static constexpr bool kBehindAll = true;  // it starts early under a kernel of its own only (sort_launch_grid)
  const uint2* kv;     // the sorted entries
  uint32_t* scratch;   // shared memory, 8 * kThreads words, free after the sort
  int4* exchange;
  unsigned* bar;
  int4* s_pref;        // shared memory [2]
  int* s_flag;         // shared memory [1]
  int* err;
  SortChunks chunks;
  int count;
  int rank, ctas, ntiles;
  unsigned arrived;    // barriers passed so far
  bool wide, none;
  __device__ __forceinline__ explicit GridCtx(int n)
      : chunks((uint32_t)n, gridDim.x, kGridT), count(n), rank(blockIdx.x), ctas(gridDim.x), arrived(0) {}
  __device__ __forceinline__ uint32_t chunk_begin() const { return chunks.begin(rank); }
  __device__ __forceinline__ uint32_t chunk_end() const { return chunks.end(rank); }
  // a tile is kGridT * kItems entries (the last one fewer), a warp takes 32 * kItems consecutive ones
  __device__ __forceinline__ uint32_t first(int t) const {
    return chunks.entry(rank, t, kGridT * kItems, (threadIdx.x >> 5) * (32 * kItems) + (threadIdx.x & 31));
  }
  __device__ __forceinline__ void get8(int j, uint2 (&e)[8]) const {
    const uint4* p = reinterpret_cast<const uint4*>(kv + j);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 x = __ldcg(p + q);
      e[2 * q] = make_uint2(x.x, x.y);
      e[2 * q + 1] = make_uint2(x.z, x.w);
    }
  }
  __device__ __forceinline__ uint2 get(int j) const { return __ldcg(kv + j); }
  __device__ __forceinline__ const uint2* publish(uint2*) { return kv; }
  struct Word {
    unsigned* at;
    __device__ __forceinline__ void add(unsigned v) const {
      asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(at), "r"(v) : "memory");
    }
    __device__ __forceinline__ unsigned load() const {
      unsigned seen;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(at) : "memory");
      return seen;
    }
    __device__ __forceinline__ bool swap(unsigned was, unsigned to) const { return atomicCAS(at, was, to) == was; }
    __device__ __forceinline__ void pause(int turn) const {
      if (turn > 4096) __nanosleep(64);
    }
  };
  // false: some CTA did not arrive within a second or two; the launch ends, its status word says so
  __device__ __forceinline__ bool barrier() {
    ++arrived;
    __syncthreads();
    if (threadIdx.x == 0) {  // (the block's stores are released with its arrival)
      Word w{bar};
      const bool ok = grid_barrier(w, arrived * (unsigned)ctas, 1 << 21);
      if (!ok && err) atomicExch(err, HB_ERR_TIMEOUT);
      *s_flag = ok;
    }
    __syncthreads();
    return *s_flag != 0;
  }
  __device__ __forceinline__ bool prefix(const int4& mine, int4& before, int4& all) {
    if (threadIdx.x == 0) __stcg(exchange + rank, mine);
    if (!barrier()) return false;
    if (threadIdx.x < 32) {
      int4 v = make_int4(0, 0, 0, 0), w = v;
      for (int c = threadIdx.x; c < ctas; c += 32) {
        const int4 x = __ldcg(exchange + c);
        if (c < rank) { v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; }
        w.x += x.x; w.y += x.y; w.z += x.z; w.w += x.w;
      }
      int4 a, t;
      a.x = __reduce_add_sync(0xffffffffu, v.x);
      a.y = __reduce_add_sync(0xffffffffu, v.y);
      a.z = __reduce_add_sync(0xffffffffu, v.z);
      a.w = __reduce_add_sync(0xffffffffu, v.w);
      t.x = __reduce_add_sync(0xffffffffu, w.x);
      t.y = __reduce_add_sync(0xffffffffu, w.y);
      t.z = __reduce_add_sync(0xffffffffu, w.z);
      t.w = __reduce_add_sync(0xffffffffu, w.w);
      if (threadIdx.x == 0) {
        s_pref[0] = a;
        s_pref[1] = t;
      }
    }
    __syncthreads();
    before = s_pref[0];
    all = s_pref[1];
    return true;
  }
};

static inline size_t sort_grid_smem_bytes(int digit) {
  const size_t bins = (size_t)1 << digit;
  return (size_t)(kGridT / 32) * bins * 6 + 2 * bins * 4 + (kGridT / 32) * 4 + 2 * sizeof(int4) + 32;
}

static __global__ void sort_grid_begin_kernel(unsigned* zero, int words) {
  begin_after_previous();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < words) zero[k] = 0u;
}

template <class Src, class Fin, int I>
__global__ void __launch_bounds__(kGridT, 1) sort_grid_kernel(Src src, Fin fin, SortGridBufs b, int max_digit, int* err) {
  wait_for_previous();
  extern __shared__ __align__(16) char smem[];
  uint16_t* wcnt = reinterpret_cast<uint16_t*>(smem);
  uint32_t* wmask = reinterpret_cast<uint32_t*>(smem + ((size_t)(kGridT / 32) << max_digit) * 2);
  uint32_t* s_base = wmask + ((kGridT / 32) << max_digit);
  uint32_t* s_tot = s_base + (1 << max_digit);
  int4* s_pref = reinterpret_cast<int4*>(s_tot + (1 << max_digit));
  uint32_t* s_warp = reinterpret_cast<uint32_t*>(s_pref + 2);
  unsigned* s_seen = s_warp + (kGridT / 32);
  int* s_flag = reinterpret_cast<int*>(s_seen + 4);
  const int n = (int)src.count();
  if (Src::kSkips && n == 0) return;
  GridCtx<I> ctx(n);
  ctx.scratch = wmask;
  ctx.exchange = b.exchange;
  ctx.bar = b.barrier;
  ctx.s_pref = s_pref;
  ctx.s_flag = s_flag;
  ctx.err = err;
  ctx.ntiles = (int)((ctx.chunks.chunk + kGridT * I - 1) / (kGridT * I));
  if (ctx.ntiles < 1) ctx.ntiles = 1;
  const int nt = ctx.ntiles;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t end = ctx.chunk_end();
  uint32_t k[I];
  uint32_t rank[(I + 1) / 2];
  SortDigits dig;
  {
    unsigned lo = 0, hi = 0;
    bool none = false;
    const bool known = sort_known_digits(src.known_bits(), max_digit, dig);
    ctx.wide = false;
    ctx.none = true;
    // (a chunk of several tiles is read again by the first pass: needed here only to find the width)
    for (int t = 0; t < nt; ++t) {
      if (nt > 1 && known) break;
      const uint32_t first = ctx.first(t);
#pragma unroll
      for (int i = 0; i < I; ++i) {
        const uint32_t j = first + i * 32;
        k[i] = kSortNone;
        if (j < end) {
          unsigned long long key;
          if (sort_load(src, j, key)) {
            k[i] = (uint32_t)key;
            lo |= (unsigned)key;
            hi |= (unsigned)(key >> 32);
          } else {
            none = true;
          }
        }
      }
    }
    if (!known) {
      lo = __reduce_or_sync(0xffffffffu, lo);
      hi = __reduce_or_sync(0xffffffffu, hi);
      none = __any_sync(0xffffffffu, none);
      if (threadIdx.x < 4) s_seen[threadIdx.x] = 0u;
      __syncthreads();
      if (lane == 0) {
        if (lo) atomicOr(s_seen, lo);
        if (hi) atomicOr(s_seen + 1, hi);
        if (none) atomicOr(s_seen + 2, 1u);
      }
      __syncthreads();
      if (threadIdx.x == 0) __stcg(reinterpret_cast<uint4*>(b.partial) + ctx.rank, make_uint4(s_seen[0], s_seen[1], s_seen[2], 0u));
      if (!ctx.barrier()) return fin.give_up(ctx, src);
      lo = hi = 0;
      unsigned nn = 0;
      for (int c = lane; c < ctx.ctas; c += 32) {
        const uint4 p = __ldcg(reinterpret_cast<const uint4*>(b.partial) + c);
        lo |= p.x; hi |= p.y; nn |= p.z;
      }
      lo = __reduce_or_sync(0xffffffffu, lo);
      hi = __reduce_or_sync(0xffffffffu, hi);
      nn = __reduce_or_sync(0xffffffffu, nn);
      dig = sort_digits(lo, hi, nn != 0, max_digit);
      ctx.wide = dig.wide;
      ctx.none = nn != 0;
    }
  }
  const uint2* in = nullptr;
  uint2* out = b.kv0;
  const int per_group = sort_group_ctas(ctx.ctas), group = ctx.rank / per_group;
  const int bins_most = 1 << max_digit;
  for (int pass = 0; pass < dig.passes; ++pass) {
    const int bit = pass * dig.width;
    const int width = dig.bits - bit < dig.width ? dig.bits - bit : dig.width;
    const int bins = 1 << width;
    const uint32_t mask = bins - 1;
    const int shift = dig.wide ? 0 : bit;
    uint16_t* wc = wcnt + warp * bins;
    // keys of a tile into k[] (already there for the first pass of a chunk of one tile)
    auto load_tile = [&](int t) {
      const uint32_t first = ctx.first(t);
      // (the keys of a pass in a loop of their own, all on their way at once: 2,000,000 ids 111.0 -> 103.6 us, 1,048,576
      // 64.5 -> 62.5; the ids four at a time 113, 68.6.  At 64 registers, of ids: 152 bytes stored and 144 loaded with 16
      // entries a thread, 24 and 16 with 8, 8 and 4 with 4, 16 and 56 with 2.)
      if (dig.wide || (!in && nt > 1)) {
#pragma unroll
        for (int i = 0; i < I; ++i) {
          const uint32_t j = first + i * 32;
          unsigned long long key;
          if (j < end) k[i] = sort_load(src, in ? __ldcg(&in[j].y) : j, key) ? (uint32_t)(dig.wide ? key >> bit : key) : kSortNone;
        }
      } else if (in) {
#pragma unroll
        for (int i = 0; i < I; ++i)
          if (first + i * 32 < end) k[i] = __ldcg(&in[first + i * 32].x);
      }
    };
    auto rank_tile = [&](int t) -> uint32_t {  // the tile's count of digit threadIdx.x
      __syncthreads();
      sort_zero_counts<kGridT>(wcnt, wmask, bins, pass == 0 && t == 0 ? (kGridT / 32) * bins : 0);
      load_tile(t);
      __syncthreads();
      sort_rank_warp<I>(k, (int)(end - ctx.first(t)), shift, width, wc, wmask + warp * bins, rank);
      __syncthreads();
      sort_scan_warps<kGridT>(wcnt, bins, s_tot);
      __syncthreads();
      return (int)threadIdx.x < bins ? s_tot[threadIdx.x] : 0u;
    };
    uint32_t mine = 0, last = 0;
    for (int t = 0; t < nt; ++t) {
      last = rank_tile(t);
      mine += last;
    }
    uint32_t* totals = b.groups + (size_t)(pass & 1) * kSortGroups * bins_most;
    if ((int)threadIdx.x < bins) {
      __stcg(b.hist + ctx.rank * bins + threadIdx.x, mine);
      if (mine) atomicAdd(totals + group * bins + threadIdx.x, mine);
    }
    if (!ctx.barrier()) return fin.give_up(ctx, src);
    // (the totals of the pass before have been read by all)
    uint32_t* next = b.groups + (size_t)((pass + 1) & 1) * kSortGroups * bins_most;
    for (int w = ctx.rank * kGridT + threadIdx.x; w < kSortGroups * bins_most; w += ctx.ctas * kGridT) __stcg(next + w, 0u);
    {
      uint32_t all = 0, pre = 0;
      if ((int)threadIdx.x < bins) {
        uint32_t x[kSortGroups], y[kSortGroups];  // all of them on their way at once
#pragma unroll
        for (int q = 0; q < kSortGroups; ++q) x[q] = __ldcg(totals + q * bins + threadIdx.x);
#pragma unroll
        for (int q = 0; q < kSortGroups; ++q) {
          const int c = group * per_group + q;
          y[q] = c < ctx.rank ? __ldcg(b.hist + c * bins + threadIdx.x) : 0u;
        }
#pragma unroll
        for (int q = 0; q < kSortGroups; ++q) {
          all += x[q];
          pre += (q < group ? x[q] : 0u) + y[q];
        }
        for (int c = group * per_group + kSortGroups; c < ctx.rank; ++c) pre += __ldcg(b.hist + c * bins + threadIdx.x);
      }
      const uint32_t start = sort_block_exscan(all, bins, s_warp);
      if ((int)threadIdx.x < bins) s_base[threadIdx.x] = start + pre;
    }
    for (int t = 0; t < nt; ++t) {
      if (nt > 1) last = rank_tile(t);
      __syncthreads();
      const uint32_t first = ctx.first(t);
#pragma unroll
      for (int i = 0; i < I; ++i) {
        const uint32_t j = first + i * 32;
        if (j < end) {
          const uint32_t d = (k[i] >> shift) & mask;
          const uint32_t to = s_base[d] + wc[d] + ((rank[i >> 1] >> (16 * (i & 1))) & 0xffffu);
          __stcg(out + to, make_uint2(k[i], in ? __ldcg(&in[j].y) : j));
        }
      }
      if (nt > 1) {
        __syncthreads();
        if ((int)threadIdx.x < bins) s_base[threadIdx.x] += last;
      }
    }
    if (!ctx.barrier()) return fin.give_up(ctx, src);
    in = out;
    out = out == b.kv0 ? b.kv1 : b.kv0;
  }
  ctx.kv = in;
  start_next();
  fin.run(ctx, src);
}

// ---- launches ------------------------------------------------------------------------------------
template <class Src, class Fin, int I>
int sort_launch_cluster(const Src& src, const Fin& fin, int ctas, cudaStream_t st) {
  const size_t smem = sort_cluster_smem_bytes(I);
  auto kernel = sort_cluster_kernel<Src, Fin, I>;
  static thread_local int ready_dev = -1;
  int dev = 0;
  HB_CUDA(cudaGetDevice(&dev));
  if (ready_dev != dev) {
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    ready_dev = dev;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kClusterT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // (HB_LAUNCH_NEXT)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = stream_captures(st) ? 1 : 2;
  HB_CUDA(cudaLaunchKernelEx(&cfg, kernel, src, fin));
  count_launch();
  return HB_OK;
}

template <class Src, class Fin, int I>
int sort_launch_grid(const Src& src, const Fin& fin, int64_t n, int max_digit, void* ws, cudaStream_t st) {
  SortGridBufs b = sort_grid_bufs(ws, n);
  // Ids of a stated width that needs no digit of 10 bits leave half of the 205 KB to the L1 cache (25 bits,
  // three digits of 9: 282,624 ids 49.3 -> 47.3 us, 2,000,000 106.6 -> 102.6).  Not below 8 bits: the
  // finish works in the words of the masks.
  SortDigits stated;
  if (sort_known_digits(src.known_bits(), max_digit, stated) && stated.width < max_digit) {
    const int digit = stated.width < 8 ? 8 : stated.width;
    if (sort_known_digits(src.known_bits(), digit, stated)) max_digit = digit;
  }
  const size_t smem = sort_grid_smem_bytes(max_digit);
  auto kernel = sort_grid_kernel<Src, Fin, I>;
  static thread_local int ready_dev = -1;
  int dev = 0;
  HB_CUDA(cudaGetDevice(&dev));
  if (ready_dev != dev) {
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sort_grid_smem_bytes(kGridDigit)));
    ready_dev = dev;
  }
  // The words that have to be zero are set by a kernel whose start, and whose successor's, overlap with the end of the
  // one before it (HB_LAUNCH_NEXT): a round of the cold cache, whose sort usually ends at once, 161.0 -> 154.7 us, sums of
  // 524,288 rows 116 -> 113.7, an update of 1,048,576 286 -> 283.5.  The sort itself lives from the end of that kernel's
  // wait on, behind all that came before (GridCtx::kBehindAll).
  const bool early = !stream_captures(st);
  const int words = (int)sort_zero_words(max_digit);
  if (early) HB_LAUNCH_NEXT(sort_grid_begin_kernel, (words + 1023) / 1024, 1024, 0, st, b.barrier, words);
  else HB_CUDA(cudaMemsetAsync(b.barrier, 0, words * sizeof(unsigned), st));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(sort_grid_ctas(n));
  cfg.blockDim = dim3(kGridT);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 2 : 1;
  HB_CUDA(cudaLaunchKernelEx(&cfg, kernel, src, fin, b, max_digit, device_error_word()));
  count_launch();
  return HB_OK;
}

// n: most entries the source can have; ws: sort_grid_bytes(n) bytes, 256-byte aligned (none needed for
// n <= kSortClusterMax)
template <class Src, class Fin>
int sort_run(const Src& src, const Fin& fin, int64_t n, void* ws, cudaStream_t st) {
  // First more CTAs, then longer chunks: what a pass issues (votes, counts, stores) is bound by one
  // SM's units, and the barrier of a larger cluster costs little more.
  if (n <= kClusterT) return sort_launch_cluster<Src, Fin, 1>(src, fin, 1, st);
  if (n <= 2 * kClusterT) return sort_launch_cluster<Src, Fin, 1>(src, fin, 2, st);
  if (n <= 4 * kClusterT) return sort_launch_cluster<Src, Fin, 1>(src, fin, 4, st);
  if (n <= 8 * kClusterT) return sort_launch_cluster<Src, Fin, 1>(src, fin, 8, st);
  if (n <= 16 * kClusterT) return sort_launch_cluster<Src, Fin, 1>(src, fin, 16, st);
  if constexpr (Fin::kOneEach) {
    set_error("a sort of %lld entries with one per thread", (long long)n);
    return HB_ERR_INVALID;
  } else {
    if (n <= 32 * kClusterT) return sort_launch_cluster<Src, Fin, 2>(src, fin, 16, st);
    if (n <= 64 * kClusterT) return sort_launch_cluster<Src, Fin, 4>(src, fin, 16, st);
    if (n <= kSortClusterMax) return sort_launch_cluster<Src, Fin, 8>(src, fin, 16, st);
    const int64_t per = ceil_div(n, sort_grid_ctas(n));
    if (per <= 2 * kGridT) return sort_launch_grid<Src, Fin, 2>(src, fin, n, kGridDigit, ws, st);
    if (per <= 4 * kGridT) return sort_launch_grid<Src, Fin, 4>(src, fin, n, kGridDigit, ws, st);
    if (per <= 8 * kGridT) return sort_launch_grid<Src, Fin, 8>(src, fin, n, kGridDigit, ws, st);
    return sort_launch_grid<Src, Fin, 16>(src, fin, n, kGridDigit, ws, st);
  }
}

#endif  // __CUDACC__

}  // namespace hb
