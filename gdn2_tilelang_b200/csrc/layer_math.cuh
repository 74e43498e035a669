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
__device__ __forceinline__ void unpack4(const Vec4<T>& v, float (&o)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = to_f32(v.x[i]);
}
// (bf16 by whole words: one instruction per element, where halves taken out first are two)
template <>
__device__ __forceinline__ void unpack4<__nv_bfloat16>(const Vec4<__nv_bfloat16>& v, float (&o)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(&v);
  o[0] = __uint_as_float(u.x << 16); o[1] = __uint_as_float(u.x & 0xffff0000u);
  o[2] = __uint_as_float(u.y << 16); o[3] = __uint_as_float(u.y & 0xffff0000u);
}
template <typename T>
__device__ __forceinline__ Vec4<T> load_raw4(const T* p) { return *reinterpret_cast<const Vec4<T>*>(p); }
template <typename T>
__device__ __forceinline__ void load4(const T* p, float (&o)[4]) { unpack4(load_raw4(p), o); }
template <typename T>
__device__ __forceinline__ void store4(T* p, const float (&o)[4]) {
  Vec4<T> v;
#pragma unroll
  for (int i = 0; i < 4; ++i) v.x[i] = from_f32<T>(o[i]);
  *reinterpret_cast<Vec4<T>*>(p) = v;
}
template <>
__device__ __forceinline__ void store4<__nv_bfloat16>(__nv_bfloat16* p, const float (&o)[4]) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

}  // namespace gdn2
