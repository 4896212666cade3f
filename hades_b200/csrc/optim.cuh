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

// W values of a row at once: 4, or 8 from rows that begin at 32 bytes (fp16: 16).  (Plain loads: what the kernel before
// has written may be read.)
template <int W> struct Floats { float x[W]; };
__device__ __forceinline__ void load_row(const float* p, Floats<4>& v) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v.x[0] = t.x; v.x[1] = t.y; v.x[2] = t.z; v.x[3] = t.w;
}
__device__ __forceinline__ void load_row(const float* p, Floats<8>& v) {
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v.x[0]), "=f"(v.x[1]), "=f"(v.x[2]), "=f"(v.x[3]), "=f"(v.x[4]), "=f"(v.x[5]), "=f"(v.x[6]), "=f"(v.x[7])
               : "l"(p));
}
__device__ __forceinline__ void load_row(const __half* p, Floats<4>& v) {
  const float4 t = EmbIO<__half>::load4(p);
  v.x[0] = t.x; v.x[1] = t.y; v.x[2] = t.z; v.x[3] = t.w;
}
__device__ __forceinline__ void load_row(const __half* p, Floats<8>& v) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const unsigned w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[k]));
    v.x[2 * k] = f.x;
    v.x[2 * k + 1] = f.y;
  }
}
__device__ __forceinline__ void store_row(float* p, const Floats<4>& v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.x[0], v.x[1], v.x[2], v.x[3]);
}
__device__ __forceinline__ void store_row(float* p, const Floats<8>& v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v.x[0]), "f"(v.x[1]), "f"(v.x[2]),
               "f"(v.x[3]), "f"(v.x[4]), "f"(v.x[5]), "f"(v.x[6]), "f"(v.x[7])
               : "memory");
}
__device__ __forceinline__ void store_row(__half* p, const Floats<4>& v) {
  EmbIO<__half>::store4(p, make_float4(v.x[0], v.x[1], v.x[2], v.x[3]));
}
__device__ __forceinline__ void store_row(__half* p, const Floats<8>& v) {
  unsigned w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const __half2 h = __floats2half2_rn(v.x[2 * k], v.x[2 * k + 1]);
    w[k] = *reinterpret_cast<const unsigned*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

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
