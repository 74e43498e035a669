// Element-wise arithmetic of the layer's kernels, and their four-element accesses.
#pragma once

#include "common.cuh"

namespace gdn2 {

// Hardware exponential, reciprocal, logarithm and reciprocal square root, one instruction each (flush-to-zero
// forms: no denormal fix-up code). A few ulp each, far inside the 16-bit storage rounding and the 2e-5 the
// float32 form is tested to; the precise division and log1pf were most of these kernels' instructions.
__device__ __forceinline__ float ex2_(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rcp_(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float lg2_(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float rsq_(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
constexpr float kLn2 = 0.6931471805599453f;
__device__ __forceinline__ float silu(float x) { return x * rcp_(1.f + ex2_(-kLog2e * x)); }
__device__ __forceinline__ float sigmoidf_(float x) { return rcp_(1.f + ex2_(-kLog2e * x)); }
__device__ __forceinline__ float softplusf_(float x) {
  const float e = ex2_(-kLog2e * fabsf(x));                // softplus(x) = max(x, 0) + log1p(exp(-|x|))
  const float l = e < 0x1p-12f ? e * (1.f - 0.5f * e) : kLn2 * lg2_(1.f + e);
  return fmaxf(x, 0.f) + l;
}
// 1 / max(sqrt(ss), 1e-12): the scale of F.normalize
__device__ __forceinline__ float inv_norm(float ss) { return rsq_(fmaxf(ss, 1e-24f)); }
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// four adjacent elements as one 8- or 16-byte access
template <typename T>
struct alignas(4 * sizeof(T)) Vec4 { T x[4]; };

template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&o)[4]) {
  const Vec4<T> v = *reinterpret_cast<const Vec4<T>*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = to_f32(v.x[i]);
}
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&o)[4]) {
  Vec4<T> v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.x[i] = from_f32<T>(o[i]);
  *reinterpret_cast<Vec4<T>*>(p) = v;
}

}  // namespace gdn2
