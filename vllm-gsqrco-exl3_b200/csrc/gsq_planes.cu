// Activations -> fp16 operand planes of the two-step product (layout: gsq_planes.cuh). Per token the power of two 2^e that
// brings its largest magnitude to [2^13, 2^14); then p = d * q * 2^e of every value, q and d those of the quantiser that
// goes with the weight type, stored as hi = fp16(p) and, with two planes, lo = fp16(p - hi): 22 bits of p, which is all
// of it where d is a half (18 bits). The reciprocal scales go behind the planes, one float per token of the padded range.
//
// One CTA per token, one warp per superblock at a time, a lane 8 values: the row is read twice, the second time from L2,
// and each value written once, a whole 128-byte line of the operand per 8 lanes. (A separate kernel for the scales and one
// CTA per slice of 64 tokens took 221 us for 8192 tokens x 17408 bf16.)
//
// Extra columns (Q4_K, Q2_K: see gsq_expand.cu), one 16-column unit per superblock: Q4_K: half(sum x) * 2^(e - 4) of the 8
// slices, then what the fp16 rounding of each slice's products lost in total / 16; Q2_K: sum of p over each of the 16
// groups / 16, as hi and lo.
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
  float* inv;
};

// bits of this lane's `v` from lanes 4 s (STEP 4) or 2 s (STEP 2), s = first .. first + 7, packed into 16 bytes
template <int STEP>
__device__ __forceinline__ uint4 gather8(uint32_t v, int first) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t a = __shfl_sync(0xFFFFFFFFu, v, STEP * (first + 2 * i)), b = __shfl_sync(0xFFFFFFFFu, v, STEP * (first + 2 * i + 1));
    w[i] = (a & 0xFFFFu) | (b << 16);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ uint32_t half_bits(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)); }

template <typename T, bool VEC, int FORM, int HU, int TP>
__global__ void __launch_bounds__(QTHREADS) planes_kernel(const T* __restrict__ x, const QuantArgs g) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __shared__ float wmax[QTHREADS / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t tok = blockIdx.x;
  const bool live = tok < g.m;
  const T* const row = x + tok * g.stride;
  float up = 0.0f, inv = 0.0f;
  if (live) {
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
  if (tid == 0) g.inv[tok] = inv;

  // where this token's chunks go
  const int nth = g.nt / 2;
  const int64_t blk = tok / g.nt;
  const int ti = (int)(tok - blk * g.nt), half = ti >= nth, tih = ti - half * nth;
  const int64_t unit = (int64_t)HU * nth * (KB * 2);               // one half of a block's k-block
  uint8_t* const b0 = g.b + ((blk * (4 * g.nsb)) * 2 + half) * unit + (tih >> 3) * 1024 + (tih & 7) * 128 + (((lane & 7) ^ (tih & 7)) << 4);
  uint8_t* const t0 = TP ? g.tb + (blk * g.nsb * 2 + half) * ((int64_t)TP * nth * 32) + (tih >> 3) * 256 + (tih & 7) * 16 : nullptr;

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
      for (int e = 0; e < 8; ++e) q[e] = amax == 0.0f ? 0.0f : roundf(div_approx(v[e], df));
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
    const float ds = d * up;
    __half2 hi[4], lo[4];
    float lost = 0.0f, total = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float p0 = ds * q[2 * e], p1 = ds * q[2 * e + 1];
      hi[e] = __floats2half2_rn(p0, p1);
      const float2 back = __half22float2(hi[e]);
      lo[e] = __floats2half2_rn(p0 - back.x, p1 - back.y);
      lost += (p0 - back.x) + (p1 - back.y);
      total += p0 + p1;
    }
    uint8_t* const dst = b0 + (int64_t)(4 * sb + (lane >> 3)) * (2 * unit);
    *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(hi);
    if constexpr (HU == 2) *reinterpret_cast<uint4*>(dst + nth * (KB * 2)) = *reinterpret_cast<const uint4*>(lo);
    if constexpr (TP == 1) {
      lost += __shfl_xor_sync(0xFFFFFFFFu, lost, 2);
      lost += __shfl_xor_sync(0xFFFFFFFFu, lost, 1);
      const uint4 c0 = gather8<4>(half_bits(sum_half * up * 0.0625f), 0), c1 = gather8<4>(half_bits(lost * 0.0625f), 0);
      uint8_t* const t = t0 + (int64_t)sb * (2 * nth * 32);
      if (lane == 0) *reinterpret_cast<uint4*>(t) = c0;
      if (lane == 1) *reinterpret_cast<uint4*>(t + 128) = c1;
    } else if constexpr (TP == 2) {
      total += __shfl_xor_sync(0xFFFFFFFFu, total, 1);
      const float s16 = total * 0.0625f;
      const __half h = __float2half_rn(s16);
      const uint32_t hb = (uint32_t)__half_as_ushort(h), lb = half_bits(s16 - __half2float(h));
      uint8_t* const t = t0 + (int64_t)sb * (2 * 2 * nth * 32);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const uint4 ch = gather8<2>(hb, 8 * c), cl = gather8<2>(lb, 8 * c);
        if (lane == 0) *reinterpret_cast<uint4*>(t + 128 * c) = ch;
        if (lane == 1) *reinterpret_cast<uint4*>(t + nth * 32 + 128 * c) = cl;
      }
    }
  }
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
      if (p.hu != 2) return GSQ_ERR_UNSUPPORTED;
      return t_planes(p.kind) == 2 ? launch_planes<T, F_Q81, 2, 2>(x, g, tokens, st) : launch_planes<T, F_Q81, 2, 0>(x, g, tokens, st);
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
