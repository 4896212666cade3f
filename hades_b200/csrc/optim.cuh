// Row update rules of the owner's sparse optimisers, shared by the stand-alone update kernels and by
// the aggregation that updates each row as soon as its sum is complete.
#pragma once

#include <cuda_fp16.h>

#include "common.cuh"

namespace hb {

struct AdamParams {
  float lr, beta1, beta2, eps, one_minus_beta1, one_minus_beta2;
};

// id -> row of this rank's shard (owner = id % stride), -1 = not ours
struct RowMap {
  int64_t offset, stride, rows;
#ifdef __CUDACC__
  __device__ __forceinline__ int64_t operator()(int64_t id) const {
    if (id < offset) return -1;
    const uint64_t d = (uint64_t)(id - offset);
    const int64_t r = stride == 1 ? (int64_t)d
                                  : (((d | (uint64_t)stride) >> 32) ? (int64_t)(d / (uint64_t)stride)
                                                                    : (int64_t)((uint32_t)d / (uint32_t)stride));
    return r < rows ? r : -1;
  }
#endif
};

#ifdef __CUDACC__

template <typename E> struct EmbIO;
template <> struct EmbIO<float> {
  static __device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
  static __device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
  static __device__ __forceinline__ float load(const float* p) { return *p; }
  static __device__ __forceinline__ void store(float* p, float v) { *p = v; }
};
template <> struct EmbIO<__half> {
  static __device__ __forceinline__ float4 load4(const __half* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const __half2 a = *reinterpret_cast<const __half2*>(&raw.x);
    const __half2 b = *reinterpret_cast<const __half2*>(&raw.y);
    const float2 fa = __half22float2(a), fb = __half22float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
  }
  static __device__ __forceinline__ void store4(__half* p, float4 v) {
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<const unsigned*>(&a);
    raw.y = *reinterpret_cast<const unsigned*>(&b);
    *reinterpret_cast<uint2*>(p) = raw;
  }
  static __device__ __forceinline__ float load(const __half* p) { return __half2float(*p); }
  static __device__ __forceinline__ void store(__half* p, float v) { *p = __float2half_rn(v); }
};

// One element of rows that are not a multiple of four columns (bias1, bias2: the bias corrections), as the
// reference divides; what the row loses.
__device__ __forceinline__ float adam_elem(float g, float& m, float& v, float bias1, float bias2,
                                           const AdamParams& p) {
  // update_mem = beta1*mem + (1-beta1)*grad; update_power = beta2*power + (1-beta2)*grad^2
  // (fused explicitly, here and below: every kernel that updates rows gives the same bits)
  m = fmaf(p.beta1, m, p.one_minus_beta1 * g);
  v = fmaf(p.beta2, v, p.one_minus_beta2 * (g * g));
  const float mc = m / bias1;
  const float vc = v / bias2;
  return p.lr * mc / (sqrtf(vc) + p.eps);  // std_values, sparse_optim.py:654-655
}

// One element of vectors.  Divisions by per-row scalars are multiplications by their reciprocals (ra, rb: 1 /
// bias correction); the element-wise division and the square root are IEEE.
__device__ __forceinline__ void adam_value(float g, float& m, float& v, float& e, float ra, float rb, const AdamParams& p) {
  m = fmaf(p.beta1, m, p.one_minus_beta1 * g);
  v = fmaf(p.beta2, v, p.one_minus_beta2 * (g * g));
  e -= p.lr * (m * ra) / (sqrtf(v * rb) + p.eps);  // sparse_optim.py:654-655
}
__device__ __forceinline__ void adagrad_value(float g, float& s, float& e, const AdamParams& p) {
  s = fmaf(g, g, s);
  e -= p.lr * g / (sqrtf(s) + p.eps);
}

#endif  // __CUDACC__

}  // namespace hb
