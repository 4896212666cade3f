// Device code that brings the lines of an index up to date after a lookup: LRU ageing of the hits,
// insertion of listed ids.  Used by kernels of its own (index.cu) and by blocks of the kernel that
// moves the rows of the same batch (runs.cu).
#pragma once

#include "index.cuh"
#include "launch.cuh"

namespace hb {

// What the insertion of listed ids needs of the index (AddLists has filled heads and next).
struct AddState {
  unsigned long long* heads;
  int32_t* batch;       // [0] batches so far, [1] blocks done, [2] batch that had long lists
  uint32_t* next;
  int64_t lines;
  int64_t* line_ids;
  int32_t* lru;
  int64_t* locs;        // [n] slots given
  uint8_t* last_writer; // nullable [n]
};

inline AddState index_add_state(const hb_index* h, uint32_t* next, int64_t* locs, uint8_t* last_writer) {
  return AddState{h->heads, h->batch + 2, next, h->lines, h->line_ids, h->lru, locs, last_writer};
}

#ifdef __CUDACC__

// The line of one set in registers.  Placement policy: src/cache/cache.h:51-88 with
// find_or_empty_entry (cache_line.h:67-78) and find_lru (cache_line.h:92-103).
struct LineState {
  int64_t lid[kWays];
  int32_t cnt[kWays];
  int last[kWays];  // which id of the batch was placed in each way last, -1 = none

  __device__ __forceinline__ void load(const int64_t* line_ids, const int32_t* lru, int64_t line) {
    const longlong2* p = reinterpret_cast<const longlong2*>(line_ids + line * kWays);
    const int4* q = reinterpret_cast<const int4*>(lru + line * kWays);
#pragma unroll
    for (int w = 0; w < kWays; w += 2) {
      const longlong2 v = p[w / 2];
      lid[w] = v.x;
      lid[w + 1] = v.y;
    }
#pragma unroll
    for (int w = 0; w < kWays; w += 4) {
      const int4 v = q[w / 4];
      cnt[w] = v.x; cnt[w + 1] = v.y; cnt[w + 2] = v.z; cnt[w + 3] = v.w;
    }
#pragma unroll
    for (int w = 0; w < kWays; ++w) last[w] = -1;
  }
  __device__ __forceinline__ void store(int64_t* line_ids, int32_t* lru, int64_t line) const {
    longlong2* p = reinterpret_cast<longlong2*>(line_ids + line * kWays);
    int4* q = reinterpret_cast<int4*>(lru + line * kWays);
#pragma unroll
    for (int w = 0; w < kWays; w += 2) p[w / 2] = make_longlong2(lid[w], lid[w + 1]);
#pragma unroll
    for (int w = 0; w < kWays; w += 4) q[w / 4] = make_int4(cnt[w], cnt[w + 1], cnt[w + 2], cnt[w + 3]);
  }
  // places the k-th id of the batch for this set; the way, -1 = refused
  __device__ __forceinline__ int place(int64_t id, int k) {
    int way = -1;
    bool exists = false;
#pragma unroll
    for (int w = 0; w < kWays; ++w) {
      if (!exists) {
        if (lid[w] == id) { way = w; exists = true; }
        else if (lid[w] == -1) way = w;  // keeps the LAST empty way
      }
    }
    if (way < 0) {
      // no empty way: least recently used = largest non-zero counter, first on ties
      int best = 0;
      int32_t tmp = cnt[0];
#pragma unroll
      for (int w = 0; w < kWays; ++w) {
        if (cnt[w] > tmp && cnt[w] != 0) { best = w; tmp = cnt[w]; }
      }
      way = tmp == 0 ? -1 : best;
    }
#pragma unroll
    for (int w = 0; w < kWays; ++w)
      if (w == way) {
        if (!exists) { lid[w] = id; cnt[w] = 0; }  // set_id zeroes the counter
        last[w] = k;
      }
    return way;
  }
  __device__ __forceinline__ bool is_last(int64_t loc, int k) const {
    if (loc < 0) return false;
    const int way = (int)(loc & (kWays - 1));
    bool yes = false;
#pragma unroll
    for (int w = 0; w < kWays; ++w)
      if (w == way) yes = last[w] == k;
    return yes;
  }
};

constexpr int kListShort = 32;  // ids of a set that are put in order in a thread's own memory

// Orders a long list (entry numbers + 1, linked through next) ascending: merge sort, bottom up.
static __device__ __noinline__ uint32_t sort_list(uint32_t head, uint32_t* next) {
  for (uint32_t size = 1;; size *= 2) {
    uint32_t p = head, tail = 0;
    head = 0;
    int merges = 0;
    while (p) {
      ++merges;
      uint32_t q = p, np = 0, nq = size;
      while (np < size && q) { ++np; q = next[q - 1]; }
      while (np || (nq && q)) {
        uint32_t e;
        if (np && (!nq || !q || p < q)) { e = p; p = next[p - 1]; --np; }
        else { e = q; q = next[q - 1]; --nq; }
        if (tail) next[tail - 1] = e; else head = e;
        tail = e;
      }
      p = q;
    }
    next[tail - 1] = 0;
    if (merges <= 1) return head;
  }
}

// where the first `cap` listed entries end (a block finds it together); the usual case: nothing to cut
template <int kBlock>
__device__ __forceinline__ int64_t add_cut(const AddEntries& e, int64_t n) {
  __shared__ long long s_cut[2];
  if (!e.total || (int64_t)*e.total <= e.cap) return n;
  __shared__ int s_warp[kBlock / 32];
  const int64_t chunks = (n + 31) / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t left = e.cap;  // listed entries still allowed
  for (int64_t c0 = 0; c0 < chunks; c0 += kBlock * 16) {
    const int64_t c = c0 + threadIdx.x * 16;
    int mine = 0;
    for (int x = 0; x < 16; ++x)
      if (c + x < chunks) mine += e.chunk_listed[c + x];
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_warp[warp] = inc;
    if (threadIdx.x == 0) s_cut[0] = -1;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kBlock / 32; ++w) {
      if (w < warp) before += s_warp[w];
      all += s_warp[w];
    }
    const int64_t first = before + inc - mine;  // listed entries of this round ahead of this thread's
    if (left >= first && left < first + mine) {
      int64_t need = left - first;
      int x = 0;
      while (need >= e.chunk_listed[c + x]) { need -= e.chunk_listed[c + x]; ++x; }
      int64_t i = (c + x) * 32;
      const int64_t end = i + 32 < n ? i + 32 : n;
      for (; i < end; ++i)
        if (e.listed[i] && need-- == 0) break;
      s_cut[0] = i;
    }
    __syncthreads();
    const int64_t cut = s_cut[0];
    if (cut >= 0) return cut;
    left -= all;
    __syncthreads();
  }
  return n;
}

// ways of a line that the batch hit: their last positions, 0 = not hit
__device__ __forceinline__ void line_marks(const unsigned long long* marks, int64_t line, uint32_t number,
                                           uint32_t (&last)[kWays]) {
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(marks + line * kWays);
#pragma unroll
  for (int w = 0; w < kWays; w += 2) {
    const ulonglong2 x = p[w / 2];
    last[w] = (uint32_t)(x.x >> 32) == number ? (uint32_t)x.x : 0u;
    last[w + 1] = (uint32_t)(x.y >> 32) == number ? (uint32_t)x.y : 0u;
  }
}

constexpr uint32_t kLongList = 0xffffffffu;  // in place of the entry: the set's list is long

// The list of entry i's set (i is in front of it) in input order into the line `st`.
template <bool DISTINCT>
__device__ __forceinline__ void walk_list(const AddEntries& e, const AddState& a, int64_t i, int64_t cut, uint32_t number,
                                          int64_t line, int64_t id, LineState& st) {
  const uint32_t behind = a.next[i];
  if (!behind) {  // the usual case: one id for the set
    const int way = i < cut ? st.place(id, 0) : -1;
    a.locs[i] = way >= 0 ? line * kWays + way : -1;
    if (a.last_writer) a.last_writer[i] = way >= 0;
    st.store(a.line_ids, a.lru, line);
    return;
  }
  // A step along the list is one trip to L2, with the id of the entry in its shadow; what the walk needs
  // again stays in the thread (reading ids in order and slots back took two more trips per entry:
  // 100,000 ids on 62,500 lists 22.9 -> 20.3 us).
  uint32_t order[kListShort];
  int64_t held[kListShort];  // the id of an entry, later its way
  order[0] = (uint32_t)i + 1u;
  held[0] = id;
  int len = 1;
  uint32_t at = behind;
  while (at && len < kListShort) {
    const uint32_t after = a.next[at - 1];
    const int64_t its = DISTINCT ? e.ids[(int64_t)at - 1] : load_settled(e.ids + (int64_t)at - 1);
    int k = len++;
    for (; k > 0 && order[k - 1] > at; --k) {
      order[k] = order[k - 1];
      held[k] = held[k - 1];
    }
    order[k] = at;
    held[k] = its;
    at = after;
  }
  if (at && DISTINCT) {
    // only ids in strides of the number of sets come here: no launch is kept ready for them
    const uint32_t first = sort_list((uint32_t)i + 1u, a.next);
    int k = 0;
    for (at = first; at; at = a.next[at - 1], ++k) {
      const int64_t x = (int64_t)at - 1;
      const int way = x < cut ? st.place(e.ids[x], k) : -1;
      a.locs[x] = way >= 0 ? line * kWays + way : -1;
    }
    if (a.last_writer) {
      k = 0;
      for (at = first; at; at = a.next[at - 1], ++k) a.last_writer[at - 1] = st.is_last(a.locs[at - 1], k);
    }
  } else if (at) {
    a.heads[line] = ((unsigned long long)number << 32) | kLongList;
    a.batch[2] = (int32_t)number;
    return;
  } else {
    for (int k = 0; k < len; ++k) {
      const int64_t x = (int64_t)order[k] - 1;
      const int way = x < cut ? st.place(held[k], k) : -1;
      a.locs[x] = way >= 0 ? line * kWays + way : -1;
      held[k] = way;
    }
    if (a.last_writer)
      for (int k = 0; k < len; ++k) a.last_writer[(int64_t)order[k] - 1] = st.is_last(held[k], k);
  }
  st.store(a.line_ids, a.lru, line);
}

// hits of run u2 at batch positions after `last`
__device__ __forceinline__ int32_t hits_after(const RunsView& v, int64_t u2, int64_t nruns, int64_t npos, int64_t last,
                                              int32_t& len) {
  const int64_t s2 = v.start(u2), e2 = v.end(u2, nruns, npos);
  len = (int32_t)(e2 - s2);
  int64_t lo = s2, hi = e2;  // first position of the run greater than `last`
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (v.pos(mid) <= last) lo = mid + 1; else hi = mid;
  }
  return (int32_t)(e2 - lo);
}

// Ageing by the run that hit `slot`: its own counter, and, from the lowest hit way, those of the ways
// that were not hit.
__device__ __forceinline__ void touch_run(const RunsView& v, const TouchMarks& t, int32_t* __restrict__ lru, int64_t u,
                                          int64_t slot, int64_t nruns, int64_t npos, uint32_t number) {
  const int64_t line = slot >> 3;
  const int way = (int)(slot & 7);
  uint32_t run[kWays];
  line_marks(t.marks, line, number, run);
  // read together with the marks: one round trip fewer for the run that ages the line
  const int4 c0 = *reinterpret_cast<const int4*>(lru + line * kWays), c1 = *reinterpret_cast<const int4*>(lru + line * kWays + 4);
  const int32_t was[kWays] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
  const int64_t end = v.end(u, nruns, npos);
  const int64_t last = v.pos(end - 1);
  int32_t total = (int32_t)(end - v.start(u)), after = 0;
  bool leader = true;
#pragma unroll
  for (int w = 0; w < kWays; ++w) {
    if (!run[w] || w == way) continue;
    int32_t len;
    after += hits_after(v, (int64_t)run[w] - 1, nruns, npos, last, len);
    total += len;
    if (w < way) leader = false;
  }
  lru[slot] = after;
  if (leader) {
#pragma unroll
    for (int w = 0; w < kWays; ++w)
      if (!run[w] && w != way) lru[line * kWays + w] = was[w] + total;
  }
}

__device__ __forceinline__ void touch_runs(const RunsView& v, const TouchMarks& t, int32_t* __restrict__ lru, int block,
                                           int blocks) {
  const uint32_t number = batch_number(t.batch);
  const int64_t nruns = v.runs();
  const int64_t npos = v.positions();
  for (int64_t u = block * (int64_t)blockDim.x + threadIdx.x; u < nruns; u += (int64_t)blocks * blockDim.x) {
    const int64_t slot = v.slot_of_run(u);
    if (slot >= 0 && slot < t.capacity) touch_run(v, t, lru, u, slot, nruns, npos, number);
  }
  batch_done(t.batch, number, blocks);
}

// Ageing of a line whose owner is about to insert into it: all its hits at once.
__device__ __forceinline__ void age_line(const RunsView& v, const TouchMarks& t, int64_t line, int64_t nruns, int64_t npos,
                                         uint32_t number, LineState& st) {
  uint32_t run[kWays];
  line_marks(t.marks, line, number, run);
  int32_t total = 0;
#pragma unroll
  for (int w = 0; w < kWays; ++w) {
    if (!run[w]) continue;
    const int64_t end = v.end((int64_t)run[w] - 1, nruns, npos);
    const int64_t last = v.pos(end - 1);
    total += (int32_t)(end - v.start((int64_t)run[w] - 1));
    int32_t after = 0, len;
    for (int x = 0; x < kWays; ++x) {
      uint32_t other = 0;
#pragma unroll
      for (int y = 0; y < kWays; ++y)
        if (y == x) other = run[y];
      if (other && x != w) after += hits_after(v, (int64_t)other - 1, nruns, npos, last, len);
    }
    st.cnt[w] = after;
  }
#pragma unroll
  for (int w = 0; w < kWays; ++w)
    if (!run[w]) st.cnt[w] += total;
}

// After the per-distinct-id lookup of a batch: hits age their lines (touch), listed misses are inserted
// (insert).  A line with both is left to the thread that inserts.
struct Maintain {
  RunsView v;          // slots by run
  TouchMarks marks;
  AddEntries e;
  AddState add;
  int touch, insert;
  int apart;           // of the blocks every other one ages and the ones between insert
  int blocks;          // that do this (an even number where they are apart)
  int spread;          // they are spread over the launch; else the first ones of it

  template <int BLOCK>
  __device__ __forceinline__ void run(int block) const {
    const uint32_t hit_number = batch_number(marks.batch), add_number = batch_number(add.batch);
    const int64_t nruns = v.runs(), npos = v.positions();
    const bool ages = touch && !(apart && (block & 1)), inserts = insert && !(apart && !(block & 1));
    const int64_t cut = inserts ? add_cut<BLOCK>(e, nruns) : 0;
    const int64_t stride = (apart ? blocks >> 1 : blocks) * (int64_t)BLOCK;
    for (int64_t u = (apart ? block >> 1 : block) * (int64_t)BLOCK + threadIdx.x; u < nruns; u += stride) {
      const int64_t slot = v.locs[u];
      if (slot >= 0) {
        if (!ages) continue;
        if (insert && (uint32_t)(add.heads[slot >> 3] >> 32) == add_number) continue;
        touch_run(v, marks, add.lru, u, slot, nruns, npos, hit_number);
      } else if (inserts && e.listed[u]) {
        const int64_t id = e.ids[u];
        const int64_t line = mod_nonneg(id, add.lines);
        if (add.heads[line] != (((unsigned long long)add_number << 32) | (unsigned long long)(u + 1))) continue;
        LineState st;
        st.load(add.line_ids, add.lru, line);
        if (touch) age_line(v, marks, line, nruns, npos, hit_number, st);
        walk_list<true>(e, add, u, cut, add_number, line, id, st);
      }
    }
    if (touch) batch_done(marks.batch, hit_number, blocks);
    if (insert) batch_done(add.batch, add_number, blocks);
  }
};

#endif  // __CUDACC__

}  // namespace hb
