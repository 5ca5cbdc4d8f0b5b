// Activations -> fp16 operand planes of the two-step product (layout: gsq_planes.cuh). For the form with integer slice sums
// (HU = 0) the quants themselves and, behind them, their d per block as fp32; else scaled products: per token the power of two 2^e that
// brings its largest magnitude to [2^13, 2^14); then p = d * q * 2^e of every value, q and d those of the quantiser that
// goes with the weight type, stored as hi = fp16(p) and, with two planes, lo = fp16(p - hi): 22 bits of p, which is all
// of it where d is a half (18 bits). The reciprocal scales go behind the planes, one float per token of the padded range.
//
// One CTA per token, one warp per superblock at a time, a lane 8 values: the row is read twice, the second time from L2,
// and each value written once, a whole 128-byte line of the operand per 8 lanes. (A separate kernel for the scales and one
// CTA per slice of 64 tokens took 221 us for 8192 tokens x 17408 bf16.)
//
// Extra columns (Q4_K, Q2_K: see gsq_expand.cu), one 16-column unit per superblock: Q4_K: half(sum x) * 2^(e - 4) of the 8
// slices, then what the fp16 rounding of each slice's products lost in total / 16; Q2_K: one unit per slice, with the sums
// of the quants of its two 16-value groups in their two columns (at most 2032: exact).
#include "gsq_planes.cuh"
#include "gsq_quant.cuh"

namespace gsq {
namespace pl {

constexpr int QTHREADS = 256;

struct QuantArgs {
  int64_t m, k, stride;
  int nt, nsb;
  uint8_t* b;
  uint8_t* tb;
  float *inv, *dx;
};

// the low 16 bits of `v` of lanes 0, 4, .. 28, packed into 16 bytes
__device__ __forceinline__ uint4 gather8(uint32_t v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t a = __shfl_sync(0xFFFFFFFFu, v, 8 * i), b = __shfl_sync(0xFFFFFFFFu, v, 8 * i + 4);
    w[i] = (a & 0xFFFFu) | (b << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint32_t half_bits(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)); }

template <typename T, bool VEC, int FORM, int HU, int TP>
__global__ void __launch_bounds__(QTHREADS) planes_kernel(const T* __restrict__ x, const QuantArgs g) {
  // Starts once every block of the expanding kernel has seen the kernels before it finish, and runs beside it: 4 to 16 us of
  // latency and reads that fit into the 40 to 75 us in which that one writes the weights. Only the last block waits for it, at
  // the end: so this grid finishes after it, and the GEMM, which waits for this grid, finds both.
  asm volatile("griddepcontrol.launch_dependents;");
  __shared__ float wmax[QTHREADS / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tok = blockIdx.x;
  const bool live = tok < g.m;
  const T* const row = x + tok * g.stride;
  float up = 0.0f, inv = 0.0f;
  if (HU > 0 && live) {
    float amax = 0.0f;
    for (int64_t c = 8 * tid; c < g.k; c += 8 * QTHREADS) {
      float v[8];
      load8<T, VEC>(row, c, v);
#pragma unroll
      for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
    if (lane == 0) wmax[warp] = amax;
    __syncthreads();
    amax = wmax[0];
#pragma unroll
    for (int w = 1; w < QTHREADS / 32; ++w) amax = fmaxf(amax, wmax[w]);
    inv = 1.0f;
    if (amax > 0.0f && amax <= 3.0e38f) {
      int e;
      frexpf(amax, &e);                        // amax = f * 2^e, f in [0.5, 1)
      inv = ldexpf(1.0f, -min(max(14 - e, -100), 100));
    }
    up = 1.0f / inv;                           // a power of two
  }
  if (HU > 0 && tid == 0) g.inv[tok] = inv;

  // where this token's chunks go
  const int nth = g.nt / 2;
  const int64_t blk = tok / g.nt;
  const int ti = (int)(tok - blk * g.nt), half = ti >= nth, tih = ti - half * nth;
  const int64_t unit = (int64_t)(HU == 2 ? 2 : 1) * nth * (KB * 2);   // one half of a block's k-block
  uint8_t* const b0 = g.b + ((blk * (4 * g.nsb)) * 2 + half) * unit + (tih >> 3) * 1024 + (tih & 7) * 128 + (((lane & 7) ^ (tih & 7)) << 4);
  uint8_t* const t0 = TP ? g.tb + (blk * g.nsb * 2 + half) * ((int64_t)(HU == 0 ? 8 : 1) * nth * 32) + (tih >> 3) * 256 + (tih & 7) * 16 : nullptr;

  for (int sb = warp; sb < g.nsb; sb += QTHREADS / 32) {
    float v[8];
    if (live) {
      load8<T, VEC>(row, (int64_t)sb * 256 + 8 * lane, v);
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.0f;
    }
    float amax = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    float d, q[8], sum_half = 0.0f;
    if constexpr (FORM == F_Q81) {
      // block_q8_1: q = round(x / d), d kept as a half
      const float df = div_approx(amax, 127.0f);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = amax == 0.0f ? 0.0f : (float)(int8_t)(int)roundf(div_approx(v[e], df));   // (as the bytes: NaN is 0)
      d = __half2float(__float2half_rn(df));
    } else {
      const float d_inv = div_approx(127.0f, amax);
#pragma unroll
      for (int e = 0; e < 8; ++e) q[e] = amax > 0.0f ? roundf(v[e] * d_inv) : 0.0f;   // (a block of zeros: 0 * inf)
      d = live ? rcp_approx(d_inv) : 0.0f;
      if constexpr (FORM == F_DS4) {
        float pa = ((v[0] + v[1]) + v[2]) + v[3];
        float pb = ((v[4] + v[5]) + v[6]) + v[7];
        pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 2);
        pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 2);
        pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 1);
        pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 1);
        const float2 ds = __half22float2(__floats2half2_rn(d, pa + pb));   // the reference keeps half2(d, sum)
        d = ds.x;
        sum_half = ds.y;
      }
    }
    if constexpr (HU == 0) {
      __half2 h[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) h[e] = __floats2half2_rn(q[2 * e], q[2 * e + 1]);
      *reinterpret_cast<uint4*>(b0 + (int64_t)(4 * sb + (lane >> 3)) * (2 * unit)) = *reinterpret_cast<const uint4*>(h);
      // (of 16 tokens, 4 i + j at place 4 j + i: a thread of the GEMM has those of one j)
      if ((lane & 3) == 0) g.dx[((blk * g.nsb + sb) * 8 + (lane >> 2)) * g.nt + (ti & ~15) + 4 * (ti & 3) + ((ti >> 2) & 3)] = live ? d : 0.0f;
      if constexpr (TP) {
        float sum = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
        // lane 2 s + c writes chunk c (8 columns) of slice s: groups 2 s and 2 s + 1 (lanes 4 s, 4 s + 2) are its columns 2 s, 2 s + 1
        const int s = (lane >> 1) & 7, c = lane & 1;
        const uint32_t hb = half_bits(sum), lo = __shfl_sync(0xFFFFFFFFu, hb, 4 * s), hi = __shfl_sync(0xFFFFFFFFu, hb, 4 * s + 2);
        const uint32_t word = lo | (hi << 16);
        const bool mine = c == (s >> 2);
        const uint4 u = make_uint4(mine && (s & 3) == 0 ? word : 0u, mine && (s & 3) == 1 ? word : 0u, mine && (s & 3) == 2 ? word : 0u,
                                   mine && (s & 3) == 3 ? word : 0u);
        if (lane < 16) *reinterpret_cast<uint4*>(t0 + (int64_t)sb * (2 * 8 * nth * 32) + s * (nth * 32) + 128 * c) = u;
      }
    } else {
      const float ds = d * up;
      __half2 hi[4], lo[4];
      float lost = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float p0 = ds * q[2 * e], p1 = ds * q[2 * e + 1];
        hi[e] = __floats2half2_rn(p0, p1);
        const float2 back = __half22float2(hi[e]);
        lo[e] = __floats2half2_rn(p0 - back.x, p1 - back.y);
        lost += (p0 - back.x) + (p1 - back.y);
      }
      uint8_t* const dst = b0 + (int64_t)(4 * sb + (lane >> 3)) * (2 * unit);
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(hi);
      if constexpr (HU == 2) *reinterpret_cast<uint4*>(dst + nth * (KB * 2)) = *reinterpret_cast<const uint4*>(lo);
      if constexpr (TP) {
        lost += __shfl_xor_sync(0xFFFFFFFFu, lost, 2);
        lost += __shfl_xor_sync(0xFFFFFFFFu, lost, 1);
        const uint4 c0 = gather8(half_bits(sum_half * up * 0.0625f)), c1 = gather8(half_bits(lost * 0.0625f));
        uint8_t* const t = t0 + (int64_t)sb * (2 * nth * 32);
        if (lane == 0) *reinterpret_cast<uint4*>(t) = c0;
        if (lane == 1) *reinterpret_cast<uint4*>(t + 128) = c1;
      }
    }
  }
  if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename T, int FORM, int HU, int TP>
static int launch_planes(const void* x, const QuantArgs& g, int64_t tokens, cudaStream_t st) {
  const bool vec = ((uintptr_t)x % 16 == 0) && ((g.stride * (int64_t)sizeof(T)) % 16 == 0);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tokens);
  cfg.blockDim = dim3(QTHREADS);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (vec) GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, planes_kernel<T, true, FORM, HU, TP>, (const T*)x, g));
  else GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, planes_kernel<T, false, FORM, HU, TP>, (const T*)x, g));
  return GSQ_OK;
}

template <typename T>
static int launch_planes_t(const Plan& p, const void* x, const QuantArgs& g, int64_t tokens, cudaStream_t st) {
  switch (form_of(p.kind)) {
    case F_DS4: return p.hu == 1 ? launch_planes<T, F_DS4, 1, 1>(x, g, tokens, st) : GSQ_ERR_UNSUPPORTED;
    case F_D4: return p.hu == 1 ? launch_planes<T, F_D4, 1, 0>(x, g, tokens, st) : launch_planes<T, F_D4, 2, 0>(x, g, tokens, st);
    default:
      if (p.hu == 2) return launch_planes<T, F_Q81, 2, 0>(x, g, tokens, st);
      return t_planes(p.kind) ? launch_planes<T, F_Q81, 0, 1>(x, g, tokens, st) : launch_planes<T, F_Q81, 0, 0>(x, g, tokens, st);
  }
}

int planes_host(const Plan& p, const void* x, int x_dtype, int64_t m, int64_t k, int64_t stride, uint8_t* scratch, cudaStream_t st) {
  QuantArgs g;
  g.m = m;
  g.k = k;
  g.stride = stride;
  g.nt = p.nt;
  g.nsb = p.nsb;
  g.b = scratch + p.b;
  g.tb = scratch + p.tb;
  g.inv = reinterpret_cast<float*>(scratch + p.inv);
  g.dx = reinterpret_cast<float*>(scratch + p.dx);
  const int64_t tokens = (int64_t)p.nt * p.n_tb;
  switch (x_dtype) {
    case GSQ_F32: return launch_planes_t<float>(p, x, g, tokens, st);
    case GSQ_F16: return launch_planes_t<__half>(p, x, g, tokens, st);
    case GSQ_BF16: return launch_planes_t<__nv_bfloat16>(p, x, g, tokens, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}

}  // namespace pl
}  // namespace gsq
