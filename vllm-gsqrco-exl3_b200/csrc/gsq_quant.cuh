// Pieces the activation quantisers share (gsq_quantize.cu, gsq_planes.cu, gsq_gemv.cu): the approximate divisions of the reference's
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

__device__ __forceinline__ uint32_t pack4(float a, float b, float c, float d) {
  // float -> int8 as the C conversion in the reference (round toward zero of an already rounded value)
  const int ia = (int)a, ib = (int)b, ic = (int)c, id = (int)d;
  return (uint32_t)(ia & 0xFF) | ((uint32_t)(ib & 0xFF) << 8) | ((uint32_t)(ic & 0xFF) << 16) | ((uint32_t)(id & 0xFF) << 24);
}

// This thread's 8 consecutive values (piece `piece` of the 32-value block its 4 adjacent lanes share) -> block_q8_1 at
// `b`. All 32 lanes of the warp must call it (shuffles); dead lanes pass zeros and live = false.
__device__ __forceinline__ void q8_1_store8(const float (&v)[8], bool live, uint8_t* b, int piece) {
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
  float s[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = v[e] + __shfl_xor_sync(0xFFFFFFFFu, v[e], 2);  // lane offset 16
#pragma unroll
  for (int e = 0; e < 8; ++e) s[e] = s[e] + __shfl_xor_sync(0xFFFFFFFFu, s[e], 1);  // lane offset 8
  const float s0 = s[0] + s[4], s1 = s[1] + s[5], s2 = s[2] + s[6], s3 = s[3] + s[7];  // offset 4
  const float sum = (s0 + s2) + (s1 + s3);                                              // offsets 2, 1
  if (!live) return;
  const float d = div_approx(amax, 127.0f);
  float q[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) q[e] = amax == 0.0f ? 0.0f : roundf(div_approx(v[e], d));
  uint32_t* q32 = reinterpret_cast<uint32_t*>(b + 4 + piece * 8);  // the quants follow the (d, sum) pair
  q32[0] = pack4(q[0], q[1], q[2], q[3]);
  q32[1] = pack4(q[4], q[5], q[6], q[7]);
  if (piece == 0) {
    *reinterpret_cast<__half2*>(b) = __floats2half2_rn(d, sum);
  }
}

}  // namespace gsq
