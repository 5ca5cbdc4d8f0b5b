// Pieces the activation quantisers share (gsq_quantize.cu, gsq_planes.cu): the approximate divisions of the reference's
// --use_fast_math build, and loads of 8 consecutive activations.
#pragma once
#include "gsq_common.cuh"

namespace gsq {

__device__ __forceinline__ float div_approx(float a, float b) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float rcp_approx(float a) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
}

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// 8 consecutive values of row `row` starting at column c (c % 8 == 0). VEC: 16-byte aligned rows.
// Loads go to L2 (ld.global.cg): launched as a programmatic dependent, this kernel can be resident while the
// kernel that writes X still runs, so X is not read-only for its lifetime and the non-coherent path is not valid.
template <typename T, bool VEC>
__device__ __forceinline__ void load8(const T* __restrict__ x, int64_t off, float (&v)[8]) {
  if constexpr (VEC && sizeof(T) == 2) {
    const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(x + off));
    const T* p = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = to_f32<T>(p[e]);
  } else if constexpr (VEC && sizeof(T) == 4) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(x + off));
    const float4 b = __ldcg(reinterpret_cast<const float4*>(x + off + 4));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = to_f32<T>(__ldcg(x + off + e));
  }
}

}  // namespace gsq
