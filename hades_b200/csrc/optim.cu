// Sparse optimiser row updates on the owning shard: Adam as the reference's
// SparseAdam.update (python/EmbCache/sparse_optim.py:590-685) and Adagrad (the
// reference has no Adagrad; the rule is the usual sparse Adagrad
// sum += g*g; emb -= lr * g / (sqrt(sum) + eps)).  State, gradient and embedding
// rows are read and written once, in one kernel; the reference moves state
// through cached fetch/set kernels and the embedding through a CPU write.
#include "launch.cuh"
#include "optim.cuh"

namespace hb {
namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ int64_t effective_n(int64_t n, const int64_t* n_dev) {
  if (!n_dev) return n;
  const int64_t d = *n_dev;
  return d < n ? d : n;
}

// A group of G lanes per row, kOptRows rows in flight per group (their loads are
// issued together, then the arithmetic and the stores follow).
constexpr int kOptRows = 2;

template <typename E, bool VEC4>
__global__ void __launch_bounds__(kBlock, 4) sparse_adam_kernel(
    const int64_t* __restrict__ ids, const float* __restrict__ grads,
    const int64_t* __restrict__ cnt, int64_t n, const int64_t* __restrict__ n_dev, int64_t dim,
    RowMap map, float* __restrict__ step, float* __restrict__ mem, float* __restrict__ power,
    E* __restrict__ emb, AdamParams p, int glog2) {
  n = effective_n(n, n_dev);
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t group = tid >> glog2;
  const int sub = (int)(tid & ((1 << glog2) - 1));
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) >> glog2;
  const int G = 1 << glog2;
  const int lane = threadIdx.x & 31;
  const int leader = lane & ~(G - 1);       // first lane of this row group
  const int64_t warp_first = group - (lane >> glog2);  // the loop bound is the same for the whole warp
  for (int64_t w0 = warp_first, i0 = group; w0 < n; w0 += ngroups * kOptRows, i0 += ngroups * kOptRows) {
    int64_t row[kOptRows];
    float bias1[kOptRows], bias2[kOptRows], c[kOptRows];
#pragma unroll
    for (int r = 0; r < kOptRows; ++r) {
      const int64_t i = i0 + r * ngroups;
      row[r] = i < n ? map(__ldg(ids + i)) : -1;
      // the per-row scalars are worked out by the group's first lane and handed round
      float b1 = 1.0f, b2 = 1.0f, cc = 1.0f;
      if (row[r] >= 0 && sub == 0) {
        // state_step = state_step + 1 (per row), sparse_optim.py:624-626
        const float t = step[row[r]] + 1.0f;
        step[row[r]] = t;  // no other lane looks at it: ids are distinct
        b1 = 1.0f - powf(p.beta1, t);
        b2 = 1.0f - powf(p.beta2, t);
        cc = cnt ? (float)__ldg(cnt + i) : 1.0f;  // grad / cnt, sparse_optim.py:608-611
      }
      bias1[r] = __shfl_sync(0xffffffffu, b1, leader);
      bias2[r] = __shfl_sync(0xffffffffu, b2, leader);
      c[r] = __shfl_sync(0xffffffffu, cc, leader);
    }
    if (VEC4) {
      for (int64_t k = sub; k < (dim >> 2); k += G) {
        float4 gg[kOptRows], mm[kOptRows], vv[kOptRows], ee[kOptRows];
#pragma unroll
        for (int r = 0; r < kOptRows; ++r)
          if (row[r] >= 0) {
            gg[r] = __ldg(reinterpret_cast<const float4*>(grads + (i0 + r * ngroups) * dim) + k);
            mm[r] = reinterpret_cast<const float4*>(mem + row[r] * dim)[k];
            vv[r] = reinterpret_cast<const float4*>(power + row[r] * dim)[k];
            ee[r] = EmbIO<E>::load4(emb + row[r] * dim + 4 * k);
          }
#pragma unroll
        for (int r = 0; r < kOptRows; ++r)
          if (row[r] >= 0) {
            if (cnt) { gg[r].x /= c[r]; gg[r].y /= c[r]; gg[r].z /= c[r]; gg[r].w /= c[r]; }
            ee[r].x -= adam_elem(gg[r].x, mm[r].x, vv[r].x, bias1[r], bias2[r], p);
            ee[r].y -= adam_elem(gg[r].y, mm[r].y, vv[r].y, bias1[r], bias2[r], p);
            ee[r].z -= adam_elem(gg[r].z, mm[r].z, vv[r].z, bias1[r], bias2[r], p);
            ee[r].w -= adam_elem(gg[r].w, mm[r].w, vv[r].w, bias1[r], bias2[r], p);
            reinterpret_cast<float4*>(mem + row[r] * dim)[k] = mm[r];
            reinterpret_cast<float4*>(power + row[r] * dim)[k] = vv[r];
            EmbIO<E>::store4(emb + row[r] * dim + 4 * k, ee[r]);
          }
      }
    } else {
      for (int64_t k = sub; k < dim; k += G) {
#pragma unroll
        for (int r = 0; r < kOptRows; ++r)
          if (row[r] >= 0) {
            float gg = __ldg(grads + (i0 + r * ngroups) * dim + k);
            if (cnt) gg /= c[r];
            float mm = mem[row[r] * dim + k], vv = power[row[r] * dim + k];
            const float upd = adam_elem(gg, mm, vv, bias1[r], bias2[r], p);
            mem[row[r] * dim + k] = mm;
            power[row[r] * dim + k] = vv;
            E* e = emb + row[r] * dim + k;
            EmbIO<E>::store(e, EmbIO<E>::load(e) - upd);
          }
      }
    }
  }
}

// The vector path of both update rules (dim % 4 == 0, 16-byte aligned rows).  A warp takes 32
// rows per round: lane l works out the per-row scalars of row l once (for Adam the two bias
// corrections, whose powf would otherwise be issued for every 16 bytes of the row), then the
// warp walks the rows, G lanes per row with W values each, taking the scalars by shuffle.
// Bound by HBM as long as the warps of an SM hide each other's arithmetic (two roots or divisions a value).  Rows of 32
// bytes a lane (rows_of_8), one in flight per lane group, against two of 16 bytes (us): Adagrad 600,000 x 64 fp16
// 128.9 -> 116.5, 524,288 x 128 228 -> 222, 40,000 x 128 23.4 -> 21.8, Adam 300,000 x 64 fp16 107.6 -> 99.4, 200,000 x 256
// 249 -> 236, 524,288 x 128 331.6 -> 330.7 (5.7 TB/s; without the arithmetic 313).  One row of 16 bytes a lane and more
// warps: 200,000 x 100 for Adam 140 -> 147.
template <typename E, bool ADAM, int W>
__global__ void __launch_bounds__(kBlock, 3) sparse_update_vec_kernel(
    const int64_t* ids, const float* grads, const int64_t* cnt, int64_t n, const int64_t* n_dev, int64_t dim,
    RowMap map, float* step, float* s0, float* s1, E* emb, AdamParams p, int glog2, int rpw) {
  begin_after_previous();
  constexpr int kFly = W == 8 ? 1 : 2;  // rows in flight per lane group
  // rpw: rows a warp takes per round (32, or fewer so that a short list still fills the GPU)
  n = effective_n(n, n_dev);
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int G = 1 << glog2, rpp = 32 >> glog2;
  const int sub = lane & (G - 1), which = lane >> glog2;
  for (int64_t base = warp * rpw; base < n; base += nwarps * rpw) {
    const int64_t i = base + lane;
    const int64_t row = (lane < rpw && i < n) ? map(ids[i]) : -1;
    float ra = 1.0f, rb = 1.0f, rc = 1.0f;
    if (row >= 0) {
      if (ADAM) {
        // state_step = state_step + 1 (per row), sparse_optim.py:624-626
        const float t = step[row] + 1.0f;
        step[row] = t;  // no other lane looks at it: ids are distinct
        ra = 1.0f / (1.0f - powf(p.beta1, t));
        rb = 1.0f / (1.0f - powf(p.beta2, t));
      }
      if (cnt) rc = 1.0f / (float)cnt[i];  // grad / cnt, sparse_optim.py:608-611
    }
    for (int q0 = 0; q0 < rpw; q0 += rpp * kFly) {
      int64_t rw[kFly];
      float a[kFly], b[kFly], c[kFly];
      const float* gp[kFly];
#pragma unroll
      for (int u = 0; u < kFly; ++u) {
        const int q = q0 + u * rpp + which;
        rw[u] = __shfl_sync(0xffffffffu, row, q & 31);
        a[u] = __shfl_sync(0xffffffffu, ra, q & 31);
        b[u] = __shfl_sync(0xffffffffu, rb, q & 31);
        c[u] = __shfl_sync(0xffffffffu, rc, q & 31);
        if (q >= rpw) rw[u] = -1;
        gp[u] = grads + (base + q) * dim;
      }
      for (int k = sub * W; k < (int)dim; k += G * W) {
        Floats<W> gg[kFly], mm[kFly], vv[kFly], ee[kFly];
#pragma unroll
        for (int u = 0; u < kFly; ++u)
          if (rw[u] >= 0) {
            const int64_t at = rw[u] * dim + k;
            load_row(gp[u] + k, gg[u]);
            load_row(s0 + at, mm[u]);
            if (ADAM) load_row(s1 + at, vv[u]);
            load_row(emb + at, ee[u]);
          }
#pragma unroll
        for (int u = 0; u < kFly; ++u)
          if (rw[u] >= 0) {
            const int64_t at = rw[u] * dim + k;
#pragma unroll
            for (int j = 0; j < W; ++j) {
              const float g = gg[u].x[j] * c[u];
              if (ADAM) adam_value(g, mm[u].x[j], vv[u].x[j], ee[u].x[j], a[u], b[u], p);
              else adagrad_value(g, mm[u].x[j], ee[u].x[j], p);
            }
            store_row(s0 + at, mm[u]);
            if (ADAM) store_row(s1 + at, vv[u]);
            store_row(emb + at, ee[u]);
          }
      }
    }
  }
}

int group_log2_for(int64_t units) {
  int g = 0;
  while ((1 << g) < units && g < 5) ++g;
  return g;
}

// rows per warp and round: 32 unless that leaves the GPU short of warps (a list of 84k rows is
// only 2.6k rounds of 32)
int rows_per_warp_for(int64_t n, int glog2) {
  const int min_rows = 32 >> glog2 > 4 ? 32 >> glog2 : 4;  // at least one pass of whole row groups
  int rpw = 32;
  while (rpw > min_rows && ceil_div(n, rpw) < (int64_t)sm_count() * 48) rpw >>= 1;
  return rpw;
}

// 32 bytes a lane (of fp16 rows 16).  Not for rows of up to 32 columns, of which a pass of a warp takes 8 or more, while
// all warps of the other form run at once (us, 32 / 16 bytes a lane: 2,000 x 32 Adam 3.82 / 3.30, 8,000 3.85 / 3.59,
// 15,000 4.35 / 5.67; 30,000 x 8 4.13 / 3.88, 60,000 4.89 / 6.82), nor for the two wide rows in flight of a short list
// for Adagrad (2,000 x 256 6.13 / 5.90, 4,000 6.41 / 6.46; 1,000 x 512 9.89 / 9.72, 2,000 10.0 / 10.2).
bool rows_of_8(int64_t n, int64_t dim, bool adam, uintptr_t state_bits, const void* emb, int emb_elem_bytes) {
  if (dim % 8 != 0 || (state_bits & 31) != 0 || ((uintptr_t)emb & (8 * emb_elem_bytes - 1)) != 0) return false;
  if (dim <= 32) return n << group_log2_for(dim / 4) > (int64_t)sm_count() * 3 * kBlock;
  return adam || dim < 256 || n * dim > (int64_t)sm_count() * 4096;
}

int grid_for_warps(int64_t n, int rpw) {
  int64_t blocks = ceil_div(ceil_div(n, rpw) * 32, kBlock);
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}

template <typename E, bool VEC4>
__global__ void __launch_bounds__(kBlock) sparse_adagrad_kernel(
    const int64_t* __restrict__ ids, const float* __restrict__ grads,
    const int64_t* __restrict__ cnt, int64_t n, const int64_t* __restrict__ n_dev, int64_t dim,
    RowMap map, float* __restrict__ state_sum, E* __restrict__ emb, float lr, float eps, int glog2) {
  n = effective_n(n, n_dev);
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t group = tid >> glog2;
  const int sub = (int)(tid & ((1 << glog2) - 1));
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) >> glog2;
  const int G = 1 << glog2;
  for (int64_t i = group; i < n; i += ngroups) {
    const int64_t row = map(__ldg(ids + i));
    if (row < 0) continue;
    const float c = cnt ? (float)__ldg(cnt + i) : 1.0f;
    const float* g = grads + i * dim;
    float* s = state_sum + row * dim;
    E* e = emb + row * dim;
    if (VEC4) {
      for (int64_t k = sub; k < (dim >> 2); k += G) {
        float4 gg = __ldg(reinterpret_cast<const float4*>(g) + k);
        if (cnt) { gg.x /= c; gg.y /= c; gg.z /= c; gg.w /= c; }
        float4 ss = reinterpret_cast<float4*>(s)[k];
        float4 ee = EmbIO<E>::load4(e + 4 * k);
        ss.x += gg.x * gg.x; ss.y += gg.y * gg.y; ss.z += gg.z * gg.z; ss.w += gg.w * gg.w;
        ee.x -= lr * gg.x / (sqrtf(ss.x) + eps);
        ee.y -= lr * gg.y / (sqrtf(ss.y) + eps);
        ee.z -= lr * gg.z / (sqrtf(ss.z) + eps);
        ee.w -= lr * gg.w / (sqrtf(ss.w) + eps);
        reinterpret_cast<float4*>(s)[k] = ss;
        EmbIO<E>::store4(e + 4 * k, ee);
      }
    } else {
      for (int64_t k = sub; k < dim; k += G) {
        float gg = __ldg(g + k);
        if (cnt) gg /= c;
        const float ss = s[k] + gg * gg;
        s[k] = ss;
        EmbIO<E>::store(e + k, EmbIO<E>::load(e + k) - lr * gg / (sqrtf(ss) + eps));
      }
    }
  }
}

int grid_for_groups(int64_t n, int glog2) {
  int64_t blocks = ceil_div(ceil_div(n, kOptRows) << glog2, kBlock);
  const int64_t cap = (int64_t)sm_count() * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (int)blocks;
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

int hb_sparse_adam(const int64_t* ids, const float* grads, const int64_t* cnt, int64_t n,
                   const int64_t* n_dev, int64_t dim, int64_t id_offset, int64_t id_stride,
                   int64_t rows, float* step, float* mem, float* power, void* emb, int emb_elem_bytes,
                   double lr, double beta1, double beta2, double eps, hb_stream_t stream) {
  HB_CHECK_ARG(n >= 0 && dim > 0 && rows > 0 && id_stride > 0, "hb_sparse_adam: bad sizes");
  HB_CHECK_ARG(emb_elem_bytes == 4 || emb_elem_bytes == 2,
               "hb_sparse_adam: embedding must be fp32 (4) or fp16 (2)");
  HB_CHECK_ARG(n == 0 || (ids && grads && step && mem && power && emb), "hb_sparse_adam: null argument");
  if (n == 0) return HB_OK;
  const AdamParams p{(float)lr, (float)beta1, (float)beta2, (float)eps, (float)(1.0 - beta1),
                     (float)(1.0 - beta2)};
  const RowMap map{id_offset, id_stride, rows};
  const uintptr_t bits = (uintptr_t)grads | (uintptr_t)mem | (uintptr_t)power;
  const bool vec4 = dim % 4 == 0 && dim < (1 << 30) && ((bits | (uintptr_t)emb) & 15) == 0;
  const bool vec8 = vec4 && rows_of_8(n, dim, true, bits, emb, emb_elem_bytes);
  const int glog2 = group_log2_for(vec8 ? dim / 8 : (vec4 ? dim / 4 : dim));
  const int grid = grid_for_groups(n, glog2);
  const int rpw = rows_per_warp_for(n, glog2);
  cudaStream_t st = (cudaStream_t)stream;
#define HB_ADAM(E, V)                                                                          \
  HB_LAUNCH((sparse_adam_kernel<E, V>), grid, kBlock, 0, st, ids, grads, cnt, n, n_dev, dim, map, \
            step, mem, power, (E*)emb, p, glog2)
#define HB_ADAM_VEC(E, W)                                                                      \
  HB_LAUNCH_NEXT((sparse_update_vec_kernel<E, true, W>), grid_for_warps(n, rpw), kBlock, 0, st, ids, grads, cnt, n, \
            n_dev, dim, map, step, mem, power, (E*)emb, p, glog2, rpw)
  if (emb_elem_bytes == 4) {
    if (vec8) HB_ADAM_VEC(float, 8); else if (vec4) HB_ADAM_VEC(float, 4); else HB_ADAM(float, false);
  } else {
    if (vec8) HB_ADAM_VEC(__half, 8); else if (vec4) HB_ADAM_VEC(__half, 4); else HB_ADAM(__half, false);
  }
#undef HB_ADAM_VEC
#undef HB_ADAM
  return HB_OK;
}

int hb_sparse_adagrad(const int64_t* ids, const float* grads, const int64_t* cnt, int64_t n,
                      const int64_t* n_dev, int64_t dim, int64_t id_offset, int64_t id_stride,
                      int64_t rows, float* state_sum, void* emb, int emb_elem_bytes, double lr,
                      double eps, hb_stream_t stream) {
  HB_CHECK_ARG(n >= 0 && dim > 0 && rows > 0 && id_stride > 0, "hb_sparse_adagrad: bad sizes");
  HB_CHECK_ARG(emb_elem_bytes == 4 || emb_elem_bytes == 2,
               "hb_sparse_adagrad: embedding must be fp32 (4) or fp16 (2)");
  HB_CHECK_ARG(n == 0 || (ids && grads && state_sum && emb), "hb_sparse_adagrad: null argument");
  if (n == 0) return HB_OK;
  const RowMap map{id_offset, id_stride, rows};
  const uintptr_t bits = (uintptr_t)grads | (uintptr_t)state_sum;
  // fp16 rows are read 8 bytes at a time on the vector path
  const bool vec4 = dim % 4 == 0 && dim < (1 << 30) && ((bits | (uintptr_t)emb) & 15) == 0;
  const bool vec8 = vec4 && rows_of_8(n, dim, false, bits, emb, emb_elem_bytes);
  const int glog2 = group_log2_for(vec8 ? dim / 8 : (vec4 ? dim / 4 : dim));
  const int grid = grid_for_groups(n, glog2);
  const int rpw = rows_per_warp_for(n, glog2);
  cudaStream_t st = (cudaStream_t)stream;
#define HB_ADAGRAD(E, V)                                                                        \
  HB_LAUNCH((sparse_adagrad_kernel<E, V>), grid, kBlock, 0, st, ids, grads, cnt, n, n_dev, dim, \
            map, state_sum, (E*)emb, (float)lr, (float)eps, glog2)
  const AdamParams p{(float)lr, 0.f, 0.f, (float)eps, 0.f, 0.f};
#define HB_ADAGRAD_VEC(E, W)                                                                    \
  HB_LAUNCH_NEXT((sparse_update_vec_kernel<E, false, W>), grid_for_warps(n, rpw), kBlock, 0, st, ids, grads, cnt, n, \
            n_dev, dim, map, nullptr, state_sum, nullptr, (E*)emb, p, glog2, rpw)
  if (emb_elem_bytes == 4) {
    if (vec8) HB_ADAGRAD_VEC(float, 8); else if (vec4) HB_ADAGRAD_VEC(float, 4); else HB_ADAGRAD(float, false);
  } else {
    if (vec8) HB_ADAGRAD_VEC(__half, 8); else if (vec4) HB_ADAGRAD_VEC(__half, 4); else HB_ADAGRAD(__half, false);
  }
#undef HB_ADAGRAD_VEC
#undef HB_ADAGRAD
  return HB_OK;
}

}  // extern "C"
