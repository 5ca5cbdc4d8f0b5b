// Host side of gsq_gemm5.cuh (products of up to 256 activation rows with exact integer slice sums), its activation
// quantiser and the sum of tiles that several CTAs have worked on.
#include "gsq_gemm5.cuh"

namespace gsq {
namespace g5 {

// Tiles that several CTAs have worked on: their parts, in CTA order. One block per tile and 8 tokens, thread = row.
template <typename T>
__global__ void __launch_bounds__(TR) sum5_kernel(const Args g, int n_cta, T* __restrict__ y) {
  asm volatile("griddepcontrol.launch_dependents;");
  const int tile = blockIdx.x, tb = tile / g.n_rt, row = (tile - tb * g.n_rt) * TR + threadIdx.x;
  auto cta_of = [&](int64_t unit) { return (int)(((unit + 1) * n_cta - 1) / g.n_units); };
  const int64_t first = (int64_t)tile * g.nsb;
  const int c0 = cta_of(first), c1 = cta_of(first + g.nsb - 1);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (c0 == c1) return;
  const bool mid = (int64_t)c0 * g.n_units / n_cta != first;     // the first CTA began before this tile: its second slot
  const int t0 = blockIdx.y * 8, tok0 = tb * g.nt;
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = 0.0f;
  for (int c = c0; c <= c1; ++c) {
    const float* p = g.part + ((2 * (int64_t)c + (c == c0 && mid ? 1 : 0)) * g.nt + t0) * TR + threadIdx.x;
#pragma unroll
    for (int i = 0; i < 8; ++i) s[i] += __ldcg(p + i * TR);
  }
  if (row >= g.nrows) return;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (tok0 + t0 + i < g.m) store_out<T>(y + (int64_t)(tok0 + t0 + i) * g.ldy + row, s[i]);
}

// X -> activation units: the arithmetic of quantize_q8_1_mmq_kernel (d = 1 / (127 / amax), fp32, or half(d), half(sum)).
// One warp per token and superblock, a lane 8 values; tokens past m are zeros.
template <typename T, bool VEC, bool DS>
__global__ void __launch_bounds__(256) units_kernel(const T* __restrict__ x, uint8_t* __restrict__ out, int64_t m, int64_t stride, int nsb, int nt) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int64_t tok = blockIdx.x;
  const int sb = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (sb >= nsb) return;
  const bool live = tok < m;
  float v[8];
  if (live) {
    load8<T, VEC>(x, tok * stride + (int64_t)sb * 256 + 8 * lane, v);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.0f;
  }
  float amax = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; ++e) amax = fmaxf(amax, fabsf(v[e]));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
  amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
  const float d_inv = div_approx(127.0f, amax);
  uint32_t q[2] = {0u, 0u};
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int qi = amax > 0.0f ? (int)roundf(v[e] * d_inv) : 0;
    q[e >> 2] |= (uint32_t)(qi & 0xFF) << (8 * (e & 3));
  }
  float d = live && amax > 0.0f ? rcp_approx(d_inv) : 0.0f;
  const int tb = (int)(tok / nt), ti = (int)(tok - (int64_t)tb * nt), s = lane >> 2, piece = lane & 3;
  uint8_t* unit = out + ((int64_t)tb * nsb + sb) * unit_bytes(DS, nt);
  *reinterpret_cast<uint2*>(unit + s * nt * 32 + (ti >> 3) * 256 + (piece >> 1) * 128 + (ti & 7) * 16 + (piece & 1) * 8) = make_uint2(q[0], q[1]);
  if constexpr (DS) {
    float pa = ((v[0] + v[1]) + v[2]) + v[3];
    float pb = ((v[4] + v[5]) + v[6]) + v[7];
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 2);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 2);
    pa += __shfl_xor_sync(0xFFFFFFFFu, pa, 1);
    pb += __shfl_xor_sync(0xFFFFFFFFu, pb, 1);
    const __half2 ds = __floats2half2_rn(d, pa + pb);   // the reference keeps half2(d, sum)
    d = __low2float(ds);
    uint8_t* su = unit + nt * 288 + (ti >> 3) * 256 + (ti & 7) * 16;
    if (piece == 0) *reinterpret_cast<__half*>(su + 2 * s) = __high2half(ds);
    if (lane == 1) *reinterpret_cast<uint4*>(su + 128) = make_uint4(0u, 0u, 0u, 0u);   // columns 8..15
  }
  if (piece == 0) reinterpret_cast<float*>(unit + nt * 256)[s * nt + ti] = d;
}

template <typename T, bool DS>
static int launch_units(const void* x, uint8_t* out, int64_t m, int64_t stride, int nsb, int nt, int tokens, cudaStream_t st) {
  const bool vec = ((uintptr_t)x % 16 == 0) && ((stride * (int64_t)sizeof(T)) % 16 == 0);
  const dim3 grid((unsigned)tokens, (unsigned)((nsb + 7) / 8));
  return vec ? launch_pdl(units_kernel<T, true, DS>, grid, 256, 0, st, (const T*)x, out, m, stride, nsb, nt)
             : launch_pdl(units_kernel<T, false, DS>, grid, 256, 0, st, (const T*)x, out, m, stride, nsb, nt);
}
template <bool DS>
static int launch_units_t(int x_dtype, const void* x, uint8_t* out, int64_t m, int64_t stride, int nsb, int nt, int tokens, cudaStream_t st) {
  switch (x_dtype) {
    case GSQ_F32: return launch_units<float, DS>(x, out, m, stride, nsb, nt, tokens, st);
    case GSQ_F16: return launch_units<__half, DS>(x, out, m, stride, nsb, nt, tokens, st);
    case GSQ_BF16: return launch_units<__nv_bfloat16, DS>(x, out, m, stride, nsb, nt, tokens, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}

constexpr int SM_COUNT = 148;   // what scratch sizes are worked out for

struct Tiles {
  int nt, n_tb, n_cta;
  size_t part, total;           // the units are at 0
};
static void tiles_of(Tiles* t, int kind, int64_t rows, int64_t m, int64_t k, int sm_count) {
  t->n_tb = (int)((m + MAX_NT - 1) / MAX_NT);
  t->nt = (int)(((m + t->n_tb - 1) / t->n_tb + 15) / 16 * 16);
  const int64_t units = (rows + TR - 1) / TR * t->n_tb * (k / 256);
  t->n_cta = (int)(units < sm_count ? units : sm_count);
  t->part = ((size_t)t->n_tb * (k / 256) * unit_bytes(kind == G5_Q4K, t->nt) + 1023) / 1024 * 1024;
  t->total = t->part + (size_t)2 * t->n_cta * t->nt * TR * 4;
}
static int kind_of(int ggml_type, int packed, int64_t rows) {
  if (ggml_type == GSQ_TYPE_IQ3_S && packed && rows % 16 == 0) return G5_IQ3S;
  if (ggml_type == GSQ_TYPE_IQ4_XS) return G5_IQ4XS;   // (one layout, whatever the flag says)
  if (ggml_type == GSQ_TYPE_Q4_K) return G5_Q4K;
  return -1;
}

int launch_iq3s(const Args& g, int n_cta, cudaStream_t st);
int launch_iq4xs(const Args& g, int n_cta, cudaStream_t st);
int launch_q4k(const Args& g, int n_cta, cudaStream_t st);
int error_flag_iq3s(int* flag);
int error_flag_iq4xs(int* flag);
int error_flag_q4k(int* flag);

}  // namespace g5

int gemm5_error_flag(int* flag) {
  int a = 0, b = 0, c = 0;
  int rc = g5::error_flag_iq3s(&a);
  if (rc == GSQ_OK) rc = g5::error_flag_iq4xs(&b);
  if (rc == GSQ_OK) rc = g5::error_flag_q4k(&c);
  *flag = a | b | c;
  return rc;
}

bool gemm5_applies(int ggml_type, int packed, int64_t rows, int64_t m) { return g5::kind_of(ggml_type, packed, rows) >= 0 && m <= 2 * g5::MAX_NT; }

size_t gemm5_scratch_bytes(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k) {
  g5::Tiles t;
  g5::tiles_of(&t, g5::kind_of(ggml_type, packed, rows), rows, m, k, g5::SM_COUNT);
  return t.total;
}

int gemm5_linear(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype, int64_t m, int64_t k,
                 int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* scratch, void* stream) {
  using namespace g5;
  const int kind = kind_of(ggml_type, packed, rows);
  if (kind < 0 || rows > INT32_MAX || k > INT32_MAX || (rows + TR - 1) / TR * 2 * (k / 256) > INT32_MAX) return GSQ_ERR_UNSUPPORTED;
  DeviceInfo di;
  int rc = device_info(&di);
  if (rc != GSQ_OK) return rc;
  Tiles t;
  tiles_of(&t, kind, rows, m, k, di.sm_count < SM_COUNT ? di.sm_count : SM_COUNT);
  const bool ds = kind == G5_Q4K;
  Args g;
  g.w = (const uint8_t*)w;
  g.row_bytes = row_bytes;
  g.nrows = (int)rows;
  g.nsb = (int)(k / 256);
  g.n_rt = (int)((rows + TR - 1) / TR);
  g.n_units = g.n_rt * t.n_tb * g.nsb;
  g.xb = (const uint8_t*)scratch;
  g.nt = t.nt;
  g.m = (int)m;
  g.b_stages = MAX_B;
  while (smem_map(kind, t.nt, g.b_stages).total > 227 * 1024) --g.b_stages;
  g.y = y;
  g.y_dtype = y_dtype;
  g.ldy = y_row_stride;
  g.part = reinterpret_cast<float*>((uint8_t*)scratch + t.part);
  cudaStream_t st = (cudaStream_t)stream;
  const int tokens = t.nt * t.n_tb;
  rc = ds ? launch_units_t<true>(x_dtype, x, (uint8_t*)scratch, m, x_row_stride, g.nsb, t.nt, tokens, st)
          : launch_units_t<false>(x_dtype, x, (uint8_t*)scratch, m, x_row_stride, g.nsb, t.nt, tokens, st);
  if (rc == GSQ_OK) rc = kind == G5_IQ3S ? launch_iq3s(g, t.n_cta, st) : kind == G5_IQ4XS ? launch_iq4xs(g, t.n_cta, st) : launch_q4k(g, t.n_cta, st);
  if (rc != GSQ_OK) return rc;
  // any tile cut between CTAs?
  bool cut = false;
  for (int c = 1; c < t.n_cta && !cut; ++c) cut = ((int64_t)c * g.n_units / t.n_cta) % g.nsb != 0;
  if (!cut) return GSQ_OK;
  const dim3 grid((unsigned)(g.n_rt * t.n_tb), (unsigned)(t.nt / 8));
  if (y_dtype == GSQ_BF16) return launch_pdl(sum5_kernel<__nv_bfloat16>, grid, TR, 0, st, g, t.n_cta, (__nv_bfloat16*)y);
  if (y_dtype == GSQ_F16) return launch_pdl(sum5_kernel<__half>, grid, TR, 0, st, g, t.n_cta, (__half*)y);
  return launch_pdl(sum5_kernel<float>, grid, TR, 0, st, g, t.n_cta, (float*)y);
}

}  // namespace gsq
