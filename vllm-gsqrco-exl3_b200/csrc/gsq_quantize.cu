// q8_1 activation quantisers for fp32 / fp16 / bf16 X (sm_100a).
//
// Same arithmetic, bit for bit, as the reference's quantize_q8_1_x and quantize_mmq_q8_1_x
// (plugin/vllm_gguf_plugin/csrc/lcpp_shim.cu:274-294, 298-355), which are built with
// --use_fast_math (plugin/setup.py:42): divisions are the approximate div.approx.ftz / rcp.approx.ftz
// forms, written out explicitly here so this file needs no global fast-math flag. The launch shape
// differs: each thread owns 8 consecutive values (one 128-bit load of 16-bit X), 4 threads share a
// 32-value block. The block sum is formed in the same order as the reference's 16,8,4,2,1
// xor-shuffle tree over one value per lane (common.cuh:468-475): lane offsets 16 and 8 become
// thread offsets 2 and 1, offsets 4,2,1 become a tree inside the thread.
#include "gsq_quant.cuh"

namespace gsq {

// MMVQ layout: block_q8_1 = half d, half sum, 32 x int8 (36 bytes).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256) quantize_q8_1_kernel(const T* __restrict__ x, uint8_t* __restrict__ out,
                                                           int64_t m, int64_t k, int64_t stride) {
  // a product kernel launched behind this one with programmatic stream serialisation may start its prologue now;
  // it waits for this grid to finish before it reads `out`
  asm volatile("griddepcontrol.launch_dependents;");
  // this kernel is itself launched with programmatic stream serialisation: it may be scheduled while the kernel
  // before it drains, and waits here until that one has finished and its writes (X, perhaps) are visible
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // one thread per 8 values
  const int64_t per_row = k >> 3;
  // whole warps stay together: k % 32 == 0 makes per_row a multiple of 4, so a 4-thread group never
  // straddles the end of the work
  const bool live = t < m * per_row;
  const int64_t row = live ? t / per_row : 0;
  const int64_t c8 = live ? t - row * per_row : 0;
  float v[8];
  if (live) {
    load8<T, VEC>(x, row * stride + c8 * 8, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  q8_1_store8(v, live, out + (row * (k >> 5) + (c8 >> 2)) * 36, (int)(c8 & 3));
}

// 8 consecutive values (a quarter of a 32-value block, 4 adjacent lanes) -> quants, the block's d and (DS) sum. All 32
// lanes of the warp must call it.
template <bool DS>
__device__ __forceinline__ void mmq_quant8(const float (&v)[8], float (&q)[8], float& d, float& sum) {
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
  sum = 0.0f;
  if constexpr (DS) {
    // the reference sums 4 values per thread, then lane offsets 4, 2, 1 over 8 threads
    float pa = ((v[0] + v[1]) + v[2]) + v[3];
    float pb = ((v[4] + v[5]) + v[6]) + v[7];
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 2);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 2);
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 1);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 1);
    sum = pa + pb;
  }
  const float d_inv = div_approx(127.0f, amax);
#pragma unroll
  for (int e = 0; e < 8; ++e) q[e] = roundf(v[e] * d_inv);
  d = rcp_approx(d_inv);
}

// 128-value blocks: 16 scale bytes + 128 x int8, block (kb, row) at (kb * m + row) * 144.
template <typename T, bool VEC, int LAYOUT>
__global__ void __launch_bounds__(256) quantize_q8_1_mmq_kernel(const T* __restrict__ x, uint8_t* __restrict__ out,
                                                               int64_t m, int64_t k, int64_t stride) {
  asm volatile("griddepcontrol.launch_dependents;");
  // this kernel is itself launched with programmatic stream serialisation: it may be scheduled while the kernel
  // before it drains, and waits here until that one has finished and its writes (X, perhaps) are visible
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t per_row = k >> 3;
  const bool live = t < m * per_row;
  const int64_t row = live ? t / per_row : 0;
  const int64_t c8 = live ? t - row * per_row : 0;
  float v[8];
  if (live) {
    load8<T, VEC>(x, row * stride + c8 * 8, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  float q[8], d, sum;
  mmq_quant8<LAYOUT == GSQ_Q8_LAYOUT_DS4>(v, q, d, sum);
  if (!live) return;
  const int64_t kb = c8 >> 4;             // 128-value block along k
  const int iqs = (int)(c8 & 15) * 8;     // value offset inside the block
  uint8_t* b = out + (kb * m + row) * 144;
  *reinterpret_cast<uint2*>(b + 16 + iqs) = make_uint2(pack4(q[0], q[1], q[2], q[3]), pack4(q[4], q[5], q[6], q[7]));
  if ((iqs & 31) == 0) {
    if constexpr (LAYOUT == GSQ_Q8_LAYOUT_DS4) {
      reinterpret_cast<__half2*>(b)[iqs >> 5] = __floats2half2_rn(d, sum);
    } else {
      reinterpret_cast<float*>(b)[iqs >> 5] = d;
    }
  }
}

// The same values in the order of the small-batch product's staging area (gsq_mmv.cuh, XL_ROWS), which then takes them in
// with bulk copies: quants [row][k] (PERM: the words of a 32-value block in the order 0 4 1 5 2 6 3 7), then d
// [k/32][mc] as floats, then (DS) the sums likewise, d and sum rounded to half as in the blocks. Columns m .. mc - 1 of
// d and sum are zeros.
template <typename T, bool VEC, bool DS, bool PERM>
__global__ void __launch_bounds__(256) quantize_q8_1_rows_kernel(const T* __restrict__ x, uint8_t* __restrict__ out,
                                                                int m, int mc, int k, int64_t stride) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int t = blockIdx.x * blockDim.x + threadIdx.x, per_row = k >> 3;
  const int row = t / per_row, c8 = t - row * per_row;
  float v[8];
  if (row < m) {
    load8<T, VEC>(x, row * stride + (int64_t)c8 * 8, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  float q[8], d, sum;
  mmq_quant8<DS>(v, q, d, sum);
  if (row >= mc) return;
  const int kb = c8 >> 2, piece = c8 & 3;
  if (row < m) {
    uint8_t* dst = out + (int64_t)row * k + kb * 32;
    const uint32_t lo = pack4(q[0], q[1], q[2], q[3]), hi = pack4(q[4], q[5], q[6], q[7]);
    if constexpr (PERM) {
      const int w = 2 * piece, s = ((w & 3) << 1) | (w >> 2);   // word w goes to slot s, word w + 1 two further
      reinterpret_cast<uint32_t*>(dst)[s] = lo;
      reinterpret_cast<uint32_t*>(dst)[s + 2] = hi;
    } else {
      *reinterpret_cast<uint2*>(dst + 8 * piece) = make_uint2(lo, hi);
    }
  } else {
    d = 0.0f;
  }
  if (piece == 0) {
    float* dd = reinterpret_cast<float*>(out + (int64_t)m * k) + (int64_t)kb * mc + row;
    if constexpr (DS) {
      const float2 h = __half22float2(__floats2half2_rn(d, sum));
      dd[0] = h.x;
      dd[(int64_t)(k >> 5) * mc] = h.y;
    } else {
      dd[0] = d;
    }
  }
}

// Activation units of the prefill GEMMs (gsq_gemm2.cu, gsq_gemm3.cu): the same quantisation as
// quantize_q8_1_mmq_kernel (32-value blocks, d = 1 / (127 / amax), D4 or DS4 scales), written in the shared-memory layout
// of the tensor-core operand so that one bulk copy brings a unit into place. A unit is one 32-value slice of a block
// of 256 tokens, [token block][superblock][slice][unit]:
//   int8 operands:  [32 token groups][2 K chunks of 16][8 tokens][16 bytes] quants       (8192 bytes)
//                   [256 tokens] float d                                                 (1024 bytes)
//                   [256 tokens] float(half(sum x))   (DS4 only)                         (1024 bytes)
//   fp16 operands (LAYOUT = Q8_TILES_H16): the same quants as fp16 numbers
//                   [32 token groups][4 K chunks of 8][8 tokens][8 fp16] quants          (16384 bytes)
//                   [256 tokens] float d                                                 (1024 bytes)
// Tokens past m (up to the end of the last block) are written as zeros. One CUDA block = 64 tokens x one slice:
// warp w holds token group w of the 64, lane = (token % 8) * 4 + 8-value piece, so a warp writes whole core matrices.
template <typename T, bool VEC, int LAYOUT>
__global__ void __launch_bounds__(256) quantize_q8_1_tiles_kernel(const T* __restrict__ x, uint8_t* __restrict__ out,
                                                                 int64_t m, int64_t k, int64_t stride) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr bool DS = LAYOUT == GSQ_Q8_LAYOUT_DS4, H16 = LAYOUT == Q8_TILES_H16;
  constexpr int UB = H16 ? 16384 + 1024 : 8192 + (DS ? 2048 : 1024);
  const int slice = blockIdx.x;              // 32-value slice along k
  const int64_t tt = blockIdx.y;             // token tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = 8 * warp + (lane >> 2), piece = lane & 3;
  const int64_t row = tt * 64 + r;
  const bool live = row < m;
  float v[8];
  if (live) {
    load8<T, VEC>(x, row * stride + (int64_t)slice * 32 + piece * 8, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
  float sum = 0.0f;
  if constexpr (DS) {
    float pa = ((v[0] + v[1]) + v[2]) + v[3];
    float pb = ((v[4] + v[5]) + v[6]) + v[7];
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 2);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 2);
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 1);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 1);
    sum = pa + pb;
  }
  const float d_inv = div_approx(127.0f, amax);
  float q[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) q[e] = live && amax > 0.0f ? roundf(v[e] * d_inv) : 0.0f;   // (a block of zeros: 0 * inf)
  const float d = live ? rcp_approx(d_inv) : 0.0f;
  const int sb = slice >> 3, s = slice & 7;
  const int rb = (int)(tt & 3) * 64 + r;   // token within its block of 256
  uint8_t* unit = out + (((tt >> 2) * (k >> 8) + sb) * 8 + s) * UB;
  if constexpr (H16) {
    // the lane's 8 values are one 16-byte row of a core matrix (integers up to 127 in magnitude: exact in fp16)
    uint8_t* dst = unit + (rb >> 3) * 512 + piece * 128 + (rb & 7) * 16;
    __half2 h[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) h[e] = __floats2half2_rn(q[2 * e], q[2 * e + 1]);
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(h);
    if (piece == 0) reinterpret_cast<float*>(unit + 16384)[rb] = d;
    return;
  }
  uint8_t* dst = unit + (rb >> 3) * 256 + (piece >> 1) * 128 + (rb & 7) * 16 + (piece & 1) * 8;
  *reinterpret_cast<uint2*>(dst) = make_uint2(pack4(q[0], q[1], q[2], q[3]), pack4(q[4], q[5], q[6], q[7]));
  if (piece == 0) {
    float* sc = reinterpret_cast<float*>(unit + 8192);
    if constexpr (DS) {
      const float2 ds = __half22float2(__floats2half2_rn(d, sum));   // the reference keeps half2(d, sum)
      sc[rb] = live ? ds.x : 0.0f;
      sc[256 + rb] = live ? ds.y : 0.0f;
    } else {
      sc[rb] = d;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// The two element-wise steps that stand in front of a quantised linear in a decoder layer, fused with its q8_1
// quantiser (block_q8_1 layout), so that the step costs one launch and the normalised / activated values never make
// a round trip through memory on their way to the quantiser. The arithmetic between the steps is the unfused one:
// every intermediate is rounded to X's type where the separate kernels would have stored it, and the quantiser part
// is q8_1_store8 above, so the q8_1 bytes equal quantising the (optional) y_out of the same call bit for bit.

template <typename T>
__device__ __forceinline__ float round_to(float v);
template <>
__device__ __forceinline__ float round_to<float>(float v) { return v; }
template <>
__device__ __forceinline__ float round_to<__half>(float v) { return __half2float(__float2half_rn(v)); }
template <>
__device__ __forceinline__ float round_to<__nv_bfloat16>(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&v)[8]) {
#pragma unroll
  for (int e = 0; e < 8; ++e) store_out<T>(p + e, v[e]);
}

// RMSNorm (optionally with the residual add in front of it) -> q8_1. One CTA per row:
//   z = T(x + residual)          (residual updated in place; z = x without one)
//   var = sum z^2 / k            (fp32: each thread adds its items in order, lanes by the 16-8-4-2-1 xor tree, the
//                                 eight warps' sums in warp order)
//   y = T(T(z * rsqrt(var + eps)) * gamma)
// which is vLLM's rms_norm / fused_add_rms_norm arithmetic (csrc/layernorm_kernels.cu: the scaled value is converted
// to the tensor's type before the multiplication by the weight), then quantised.
template <typename T>
__global__ void __launch_bounds__(256) rmsnorm_q8_1_kernel(const T* __restrict__ x, int64_t stride, T* __restrict__ residual,
                                                          const T* __restrict__ gamma, float eps, uint8_t* __restrict__ out,
                                                          T* __restrict__ y_out, int64_t k) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  extern __shared__ float zrow[];          // the row after the residual add, as fp32
  __shared__ float wsum[8];
  const int64_t row = blockIdx.x;
  const int tid = threadIdx.x, per_row = (int)(k >> 3);
  float ss = 0.0f;
  for (int it = tid; it < per_row; it += 256) {
    float v[8];
    load8<T, false>(x, row * stride + (int64_t)it * 8, v);
    if (residual) {
      float r[8];
      load8<T, false>(residual, row * k + (int64_t)it * 8, r);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = round_to<T>(v[e] + r[e]);
      store8<T>(residual + row * k + (int64_t)it * 8, v);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      zrow[it * 8 + e] = v[e];
      ss = fmaf(v[e], v[e], ss);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if ((tid & 31) == 0) wsum[tid >> 5] = ss;
  __syncthreads();
  float tot = wsum[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) tot += wsum[w];
  const float rs = rsqrtf(tot / (float)k + eps);
  // whole warps pass q8_1_store8 together: the loop bound is rounded up to the warp
  for (int it0 = 0; it0 < per_row; it0 += 256) {
    const int it = it0 + tid;
    const bool live = it < per_row;
    float v[8];
    if (live) {
      float g[8];
      load8<T, false>(gamma, (int64_t)it * 8, g);
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = round_to<T>(round_to<T>(zrow[it * 8 + e] * rs) * g[e]);
      if (y_out) store8<T>(y_out + row * k + (int64_t)it * 8, v);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.0f;
    }
    q8_1_store8(v, live, out + (row * (k >> 5) + (it >> 2)) * 36, it & 3);
  }
}

// SwiGLU -> q8_1: gate_up [m, 2 * inter] (gate = the first `inter` columns, up = the rest), as vLLM's silu_and_mul
// (csrc/activation_kernels.cu): y = T(g / (1 + exp(-g))) * u in T arithmetic, then quantised over the `inter` columns.
template <typename T>
__global__ void __launch_bounds__(256) silu_mul_q8_1_kernel(const T* __restrict__ gu, int64_t stride, uint8_t* __restrict__ out,
                                                           T* __restrict__ y_out, int64_t m, int64_t inter) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // one thread per 8 values
  const int64_t per_row = inter >> 3;
  const bool live = t < m * per_row;
  const int64_t row = live ? t / per_row : 0;
  const int64_t c8 = live ? t - row * per_row : 0;
  float v[8];
  if (live) {
    float g[8], u[8];
    load8<T, false>(gu, row * stride + c8 * 8, g);
    load8<T, false>(gu, row * stride + inter + c8 * 8, u);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = round_to<T>(round_to<T>(g[e] / (1.0f + expf(-g[e]))) * u[e]);
    if (y_out) store8<T>(y_out + row * inter + c8 * 8, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  q8_1_store8(v, live, out + (row * (inter >> 5) + (c8 >> 2)) * 36, (int)(c8 & 3));
}

// launch with programmatic stream serialisation (see griddepcontrol.wait in the kernels)
template <typename... KArgs, typename... Args>
static int launch_pdl(void (*kern)(KArgs...), unsigned grid, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
  return GSQ_OK;
}

template <typename T>
static int launch_q8_1(const void* x, int64_t m, int64_t k, int64_t stride, void* out, cudaStream_t st) {
  const int64_t threads = m * (k >> 3);
  if (threads == 0) return GSQ_OK;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  const bool vec = ((uintptr_t)x % 16 == 0) && ((stride * (int64_t)sizeof(T)) % 16 == 0);
  return vec ? launch_pdl(quantize_q8_1_kernel<T, true>, grid, st, (const T*)x, (uint8_t*)out, m, k, stride)
             : launch_pdl(quantize_q8_1_kernel<T, false>, grid, st, (const T*)x, (uint8_t*)out, m, k, stride);
}

template <typename T, int LAYOUT>
static int launch_q8_1_mmq(const void* x, int64_t m, int64_t k, int64_t stride, void* out, cudaStream_t st) {
  const int64_t threads = m * (k >> 3);
  if (threads == 0) return GSQ_OK;
  const unsigned grid = (unsigned)((threads + 255) / 256);
  const bool vec = ((uintptr_t)x % 16 == 0) && ((stride * (int64_t)sizeof(T)) % 16 == 0);
  return vec ? launch_pdl(quantize_q8_1_mmq_kernel<T, true, LAYOUT>, grid, st, (const T*)x, (uint8_t*)out, m, k, stride)
             : launch_pdl(quantize_q8_1_mmq_kernel<T, false, LAYOUT>, grid, st, (const T*)x, (uint8_t*)out, m, k, stride);
}

template <typename T, int LAYOUT>
static int launch_q8_1_tiles(const void* x, int64_t m, int64_t k, int64_t stride, void* out, cudaStream_t st) {
  if (m == 0) return GSQ_OK;
  const bool vec = ((uintptr_t)x % 16 == 0) && ((stride * (int64_t)sizeof(T)) % 16 == 0);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(k >> 5), (unsigned)((m + 255) / 256 * 4));   // whole blocks of 256 tokens
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (vec) {
    GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, quantize_q8_1_tiles_kernel<T, true, LAYOUT>, (const T*)x, (uint8_t*)out, m, k, stride));
  } else {
    GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, quantize_q8_1_tiles_kernel<T, false, LAYOUT>, (const T*)x, (uint8_t*)out, m, k, stride));
  }
  return GSQ_OK;
}

template <typename T, bool DS, bool PERM>
static int launch_q8_1_rows(const void* x, int64_t m, int mc, int64_t k, int64_t stride, void* out, cudaStream_t st) {
  const unsigned grid = (unsigned)((mc * (k >> 3) + 255) / 256);
  const bool vec = ((uintptr_t)x % 16 == 0) && ((stride * (int64_t)sizeof(T)) % 16 == 0);
  return vec ? launch_pdl(quantize_q8_1_rows_kernel<T, true, DS, PERM>, grid, st, (const T*)x, (uint8_t*)out, (int)m, mc, (int)k, stride)
             : launch_pdl(quantize_q8_1_rows_kernel<T, false, DS, PERM>, grid, st, (const T*)x, (uint8_t*)out, (int)m, mc, (int)k, stride);
}
// x [m, k] -> the small-batch product's staging order (see quantize_q8_1_rows_kernel); m <= mc <= 48, k % 256 == 0.
int quantize_rows_host(const void* x, int x_dtype, int64_t m, int mc, int64_t k, int64_t stride, int ggml_type, void* out, void* stream) {
  if (m <= 0 || m > mc || mc > 48 || k <= 0 || k % 256 != 0 || k > (1 << 24) || !x || !out) return GSQ_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
#define GSQ_ROWS_CASE(T)                                                                               \
  return ggml_type == GSQ_TYPE_Q4_K     ? launch_q8_1_rows<T, true, false>(x, m, mc, k, stride, out, st) \
         : ggml_type == GSQ_TYPE_IQ4_XS ? launch_q8_1_rows<T, false, true>(x, m, mc, k, stride, out, st) \
                                        : launch_q8_1_rows<T, false, false>(x, m, mc, k, stride, out, st)
  switch (x_dtype) {
    case GSQ_F32: GSQ_ROWS_CASE(float);
    case GSQ_F16: GSQ_ROWS_CASE(__half);
    case GSQ_BF16: GSQ_ROWS_CASE(__nv_bfloat16);
    default: return GSQ_ERR_UNSUPPORTED;
  }
#undef GSQ_ROWS_CASE
}

// x [m, k] -> activation tiles for the prefill GEMM (see quantize_q8_1_tiles_kernel); k % 256 == 0.
int quantize_tiles_host(const void* x, int x_dtype, int64_t m, int64_t k, int64_t stride, int layout, void* out, void* stream) {
  if (m < 0 || k <= 0 || k % 256 != 0 || (m > 0 && (!x || !out)) || (m + 255) / 256 * 4 > 65535) return GSQ_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
#define GSQ_TILES_CASE(T)                                                                                  \
  return layout == Q8_TILES_H16      ? launch_q8_1_tiles<T, Q8_TILES_H16>(x, m, k, stride, out, st)     \
         : layout == GSQ_Q8_LAYOUT_D4 ? launch_q8_1_tiles<T, GSQ_Q8_LAYOUT_D4>(x, m, k, stride, out, st) \
                                      : launch_q8_1_tiles<T, GSQ_Q8_LAYOUT_DS4>(x, m, k, stride, out, st)
  switch (x_dtype) {
    case GSQ_F32: GSQ_TILES_CASE(float);
    case GSQ_F16: GSQ_TILES_CASE(__half);
    case GSQ_BF16: GSQ_TILES_CASE(__nv_bfloat16);
    default: return GSQ_ERR_UNSUPPORTED;
  }
#undef GSQ_TILES_CASE
}

}  // namespace gsq

extern "C" int gsq_quantize_q8_1(const void* x, int x_dtype, int64_t m, int64_t k, int64_t x_row_stride, void* out,
                                 void* stream) {
  if (m < 0 || k <= 0 || k % 32 != 0 || (m > 0 && (!x || !out))) return GSQ_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  switch (x_dtype) {
    case GSQ_F32: return gsq::launch_q8_1<float>(x, m, k, x_row_stride, out, st);
    case GSQ_F16: return gsq::launch_q8_1<__half>(x, m, k, x_row_stride, out, st);
    case GSQ_BF16: return gsq::launch_q8_1<__nv_bfloat16>(x, m, k, x_row_stride, out, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}

extern "C" int gsq_quantize_q8_1_mmq(const void* x, int x_dtype, int64_t m, int64_t k, int64_t x_row_stride,
                                     int layout, void* out, void* stream) {
  if (m < 0 || k <= 0 || k % 128 != 0 || (m > 0 && (!x || !out))) return GSQ_ERR_UNSUPPORTED;
  if (layout != GSQ_Q8_LAYOUT_D4 && layout != GSQ_Q8_LAYOUT_DS4) return GSQ_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
#define GSQ_MMQ_CASE(T)                                                                                   \
  return layout == GSQ_Q8_LAYOUT_D4 ? gsq::launch_q8_1_mmq<T, GSQ_Q8_LAYOUT_D4>(x, m, k, x_row_stride, out, st) \
                                    : gsq::launch_q8_1_mmq<T, GSQ_Q8_LAYOUT_DS4>(x, m, k, x_row_stride, out, st)
  switch (x_dtype) {
    case GSQ_F32: GSQ_MMQ_CASE(float);
    case GSQ_F16: GSQ_MMQ_CASE(__half);
    case GSQ_BF16: GSQ_MMQ_CASE(__nv_bfloat16);
    default: return GSQ_ERR_UNSUPPORTED;
  }
#undef GSQ_MMQ_CASE
}

namespace gsq {

template <typename T>
static int launch_rmsnorm_q8_1(const void* x, int64_t m, int64_t k, int64_t stride, void* residual, const void* gamma, float eps,
                               void* out, void* y_out, cudaStream_t st) {
  static std::atomic<bool> configured[64];
  int dev = 0;
  GSQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return GSQ_ERR_UNSUPPORTED;
  if (!configured[dev]) {
    GSQ_CUDA_TRY(cudaFuncSetAttribute(rmsnorm_q8_1_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
    configured[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)m);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = (size_t)k * 4;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, rmsnorm_q8_1_kernel<T>, (const T*)x, stride, (T*)residual, (const T*)gamma, eps,
                                  (uint8_t*)out, (T*)y_out, k));
  return GSQ_OK;
}

}  // namespace gsq

extern "C" int gsq_rmsnorm_quantize_q8_1(const void* x, int x_dtype, int64_t m, int64_t k, int64_t x_row_stride,
                                         void* residual, const void* gamma, float eps, void* out_q8, void* y_out,
                                         void* stream) {
  if (m == 0) return GSQ_OK;
  if (m < 0 || m > 65535 || k <= 0 || k % 32 != 0 || k > 40960 || !x || !gamma || !out_q8) return GSQ_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  switch (x_dtype) {
    case GSQ_F32: return gsq::launch_rmsnorm_q8_1<float>(x, m, k, x_row_stride, residual, gamma, eps, out_q8, y_out, st);
    case GSQ_F16: return gsq::launch_rmsnorm_q8_1<__half>(x, m, k, x_row_stride, residual, gamma, eps, out_q8, y_out, st);
    case GSQ_BF16: return gsq::launch_rmsnorm_q8_1<__nv_bfloat16>(x, m, k, x_row_stride, residual, gamma, eps, out_q8, y_out, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}

extern "C" int gsq_silu_mul_quantize_q8_1(const void* gate_up, int x_dtype, int64_t m, int64_t inter, int64_t row_stride,
                                          void* out_q8, void* y_out, void* stream) {
  if (m == 0) return GSQ_OK;
  if (m < 0 || inter <= 0 || inter % 32 != 0 || !gate_up || !out_q8) return GSQ_ERR_UNSUPPORTED;
  const int64_t threads = m * (inter >> 3);
  const unsigned grid = (unsigned)((threads + 255) / 256);
  cudaStream_t st = (cudaStream_t)stream;
  switch (x_dtype) {
    case GSQ_F32:
      return gsq::launch_pdl(gsq::silu_mul_q8_1_kernel<float>, grid, st, (const float*)gate_up, row_stride, (uint8_t*)out_q8,
                             (float*)y_out, m, inter);
    case GSQ_F16:
      return gsq::launch_pdl(gsq::silu_mul_q8_1_kernel<__half>, grid, st, (const __half*)gate_up, row_stride, (uint8_t*)out_q8,
                             (__half*)y_out, m, inter);
    case GSQ_BF16:
      return gsq::launch_pdl(gsq::silu_mul_q8_1_kernel<__nv_bfloat16>, grid, st, (const __nv_bfloat16*)gate_up, row_stride,
                             (uint8_t*)out_q8, (__nv_bfloat16*)y_out, m, inter);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}
