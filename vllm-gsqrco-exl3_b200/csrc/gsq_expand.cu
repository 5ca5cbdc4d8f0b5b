// Quantised weight rows -> fp16 tensor-core operand tiles in global memory (layout: gsq_planes.cuh), the first step of the
// two-step product. Each weight is decoded ONCE per product, not once per block of 256 tokens, and the GEMM that follows
// (gsq_gemm4.cu) has no decoding beside its multiplications: the fused kernel it replaces spent the shared-memory
// bandwidth of its SM on decoded-tile stores and codebook gathers and reached 0.40 of the fp16 rate.
//
// What goes into the operand is the integer sub-scale times the integer value, exact in fp16 (Q6_K: as a pair; IQ4_XS:
// rounded once above 2048; Q4_K with sigma != d: see q4k_sigma), and one fp32 factor per row and superblock beside it.
//
// Bound: the write of 2 bytes per weight (HBM, or L2 where it fits) plus the read of the quantised bytes. A CTA takes 64
// rows x one superblock at a time: raw bytes through registers into shared memory one item ahead, decoded into the
// operand's own byte order in shared memory, written with 8 KB bulk stores. Several CTAs per SM overlap one's loads with
// another's decoding.
#include <cuda_fp16.h>

#include "gsq_f1_codec.cuh"
#include "gsq_planes.cuh"
#include "gsq_tables.h"
#include "gsq_tc.cuh"

namespace gsq {
namespace pl {

using tc::prmt;

static __device__ const uint32_t g_x_iq3s_grid[512] = GSQ_IQ3S_GRID_INIT;
static __constant__ __align__(16) int8_t c_x_iq4nl[16] = GSQ_IQ4NL_VALUES_INIT;

struct ExpandArgs {
  const uint8_t* w;
  int64_t row_bytes;
  int nrows;      // rows of this call (tiles past the last row are written as zeros)
  int n_items;    // half row tiles x superblocks
  int nsb;
  uint8_t* a;     // [row tile][k-block][plane][16 KB]
  float *dw, *dm; // [row tile][superblock][128]
  uint8_t* ta;    // [row tile][superblock][4096]
};

constexpr int XROWS = 64, XTHREADS = 256;
constexpr int GRID_REP = 4;                    // replicas of the IQ3_S codebook, (g, -g) each

__host__ __device__ constexpr int x_block(int kind) {
  return kind == K_Q4K ? 144 : kind == K_IQ4XS ? 136 : kind == K_IQ3S_PACKED || kind == K_IQ3S ? 110 : kind == K_Q6K_PACKED || kind == K_Q6K ? 210
         : kind == K_Q2K ? 84 : kind == K_IQ2XXS ? 66 : kind == K_IQ2XS ? 74 : kind == K_IQ2S ? 82 : kind == K_IQ3XXS ? 98 : 56;
}
__host__ __device__ constexpr bool x_packed(int kind) { return kind == K_IQ3S_PACKED || kind == K_Q6K_PACKED; }
// bytes of one load and bytes of a row's (or 16-row record's) place in shared memory: rows an odd number of words (or of
// 16-byte pieces) apart, so that threads of different rows hit different banks
__host__ __device__ constexpr int x_unit(int kind) { return x_packed(kind) || kind == K_Q4K ? 16 : kind == K_IQ4XS ? 8 : 2; }
__host__ __device__ constexpr int x_segment(int kind) { return x_packed(kind) ? 16 * x_block(kind) : x_block(kind); }
__host__ __device__ constexpr int x_stride(int kind) {
  return x_unit(kind) != 2 ? x_segment(kind) : ((x_block(kind) + 3) / 4 % 2 ? (x_block(kind) + 3) / 4 * 4 : (x_block(kind) + 3) / 4 * 4 + 4);
}
__host__ __device__ constexpr int x_segments(int kind) { return x_packed(kind) ? XROWS / 16 : XROWS; }
__host__ __device__ constexpr int x_raw(int kind) { return (x_segments(kind) * x_stride(kind) + 15) / 16 * 16; }
__host__ __device__ constexpr int x_out(int kind) { return a_planes(kind) * XROWS * 256 * 2; }
__host__ __device__ constexpr int x_table(int kind) { return kind == K_IQ3S_PACKED || kind == K_IQ3S ? 512 * 8 * GRID_REP : 0; }
__host__ __device__ constexpr int x_smem(int kind) { return x_out(kind) + x_table(kind) + 2 * x_raw(kind); }

template <int UNIT>
struct Unit { using T = uint4; };
template <>
struct Unit<8> { using T = uint2; };
template <>
struct Unit<2> { using T = uint16_t; };

__device__ __forceinline__ uint32_t x_hfma2(uint32_t a, __half2 b, __half2 c) {
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&a), b, c);
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }

// byte of chunk c (8 values) of row r of a k-block's half tile (64 rows) in the out buffer
__device__ __forceinline__ uint32_t out_at(int kb, int plane, int planes, int r, int c) {
  return (uint32_t)((kb * planes + plane) * (XROWS * KB * 2) + (r >> 3) * 1024 + (r & 7) * 128 + ((c ^ (r & 7)) << 4));
}
// 4 values as bytes biased by 128 -> value * sub: a byte under the high byte 0x64 is the fp16 number 1152 + value, and
// (1152 + value) * sub - 1152 * sub in one fused multiply-add is value * sub with one rounding (|sub| <= 56: the constant
// is exact)
struct Sub {
  __half2 s, n;
  __device__ __forceinline__ explicit Sub(int sub) {
    const __half h = __int2half_rn(sub);
    s = __half2half2(h);
    n = __half2half2(__hmul(__float2half_rn(-1152.0f), h));
  }
};
__device__ __forceinline__ uint2 scale4(uint32_t v, const Sub& f) {
  return make_uint2(x_hfma2(prmt(v, 0x64646464u, 0x4140u), f.s, f.n), x_hfma2(prmt(v, 0x64646464u, 0x4342u), f.s, f.n));
}
__device__ __forceinline__ uint4 scale8(uint32_t v0, uint32_t v1, const Sub& f) {
  const uint2 a = scale4(v0, f), b = scale4(v1, f);
  return make_uint4(a.x, a.y, b.x, b.y);
}
// the same for Q6_K (|sub| up to 128, so the product needs two planes): value exact, hi = fp16(value * sub), lo = the rest
__device__ __forceinline__ void scale4_pair(uint32_t v, __half2 sc, uint2& hi, uint2& lo) {
  const __half2 bias = __float2half2_rn(-1152.0f);
  uint32_t h[2], l[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const uint32_t b = prmt(v, 0x64646464u, i ? 0x4342u : 0x4140u);
    const __half2 x = __hadd2(*reinterpret_cast<const __half2*>(&b), bias);
    const __half2 p = __hmul2(x, sc);
    h[i] = bits(p);
    l[i] = bits(__hfma2(x, sc, __hneg2(p)));
  }
  hi = make_uint2(h[0], h[1]);
  lo = make_uint2(l[0], l[1]);
}

// ---- per kind: thread (row r of 64, k-block kb) or, for the packed kinds, (warp, lane) -> operand bytes; `s` = the row's
// block (or the records) in shared memory, `grow` = row of the row tile for dw / ta. Returns through pointers only.

__device__ __forceinline__ void x_iq4_lookup(uint32_t v, const uint32_t (&tb)[4], uint32_t& lo, uint32_t& hi) {
  // (a byte permute reads the low 16 bits of its selector, so the upper four nibbles' selectors are one shift away)
  const uint32_t s01 = v & 0x77777777u, s23 = s01 >> 16;
  const uint32_t pick01 = ((v >> 1) & 0x44444444u) | 0x32103210u, pick23 = pick01 >> 16;
  const uint32_t r01 = prmt(prmt(tb[0], tb[1], s01), prmt(tb[2], tb[3], s01), pick01);
  const uint32_t r23 = prmt(prmt(tb[0], tb[1], s23), prmt(tb[2], tb[3], s23), pick23);
  lo = prmt(r01, r23, 0x6420u);
  hi = prmt(r01, r23, 0x7531u);
}

__device__ __forceinline__ void x_iq4xs(const uint8_t* s, uint8_t* out, int r, int kb, float* dw) {
  const uint2 hdr = *reinterpret_cast<const uint2*>(s);
  uint32_t tb[4];
  const uint32_t* tw = reinterpret_cast<const uint32_t*>(c_x_iq4nl);
#pragma unroll
  for (int e = 0; e < 4; ++e) tb[e] = tw[e] ^ 0x80808080u;
#pragma unroll
  for (int sl = 0; sl < 2; ++sl) {
    const int p = 2 * kb + sl;
    const uint2 qa = *reinterpret_cast<const uint2*>(s + 8 + 16 * p), qb = *reinterpret_cast<const uint2*>(s + 16 + 16 * p);
    const uint32_t v[4] = {qa.x, qa.y, qb.x, qb.y};
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) x_iq4_lookup(v[e], tb, lo[e], hi[e]);
    const Sub f((int)(((hdr.y >> (4 * p)) & 0xFu) | (((hdr.x >> (16 + 2 * p)) & 3u) << 4)) - 32);
    *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl)) = scale8(lo[0], lo[1], f);
    *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + 1)) = scale8(lo[2], lo[3], f);
    *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + 2)) = scale8(hi[0], hi[1], f);
    *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + 3)) = scale8(hi[2], hi[3], f);
  }
  if (kb == 0) *dw = h2f(hdr.x);
}

// The scale of a superblock with minimums: normally d itself, so that the operand holds the integers sc * q exactly; where
// dmin is more than 64 times d (or d is zero), dmin / 64, so that the minimum terms -(dmin / sigma) * m * 16 stay inside
// fp16 (at most 64 * 63 * 16).
__device__ __forceinline__ float sigma_of(uint32_t d_dmin) {
  const float d = h2f(d_dmin), dm = h2f(d_dmin >> 16);
  const float sigma = fabsf(dm) > 64.0f * fabsf(d) ? fabsf(dm) * (1.0f / 64.0f) : d;
  return sigma == 0.0f ? 1.0f : sigma;
}
__device__ __forceinline__ void x_q4k_scale_min(const uint4& hdr, int jj, uint32_t& sc, uint32_t& mn) {
  const uint32_t selh = (jj & 1) ? 0x4432u : 0x4410u;
  const uint32_t A = prmt(hdr.y, 0u, selh), B = prmt(hdr.z, 0u, selh), C = prmt(hdr.w, 0u, selh);
  sc = jj < 2 ? (A & 0x3F3Fu) : ((C & 0x0F0Fu) | ((A & 0xC0C0u) >> 2));
  mn = jj < 2 ? (B & 0x3F3Fu) : (((C >> 4) & 0x0F0Fu) | ((B & 0xC0C0u) >> 2));
}

// Q4_K: k-block kb = 32 bytes of quants, low nibbles slice 2 kb, high nibbles slice 2 kb + 1; (1024 + q) * f - 1024 * f.
// Extra columns, chunk 0: -(dmin / sigma) * m_s * 16, against half(sum x) * 2^(e - 4): the minimum term; chunk 1:
// 8 * (d / sigma) * sc_s * 16, against what the fp16 rounding of the slice's products lost in total / 16: the quants
// 0..15 act on the rounding errors as 8 + (q - 8), and this gives the 8's share back, so that only the centred part of
// the weights sees them.
__device__ __forceinline__ void x_q4k(const uint8_t* s, uint8_t* out, int r, int kb, float* dw, uint8_t* ta) {
  const uint4 hdr = *reinterpret_cast<const uint4*>(s);
  const float sigma = sigma_of(hdr.x), ratio = h2f(hdr.x) / sigma;
  uint32_t sc, mn;
  x_q4k_scale_min(hdr, kb, sc, mn);
  const uint4 va = *reinterpret_cast<const uint4*>(s + 16 + 32 * kb), vb = *reinterpret_cast<const uint4*>(s + 32 + 32 * kb);
  const uint32_t w[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
#pragma unroll
  for (int sl = 0; sl < 2; ++sl) {
    const __half fh = __float2half_rn(ratio * (float)((sc >> (8 * sl)) & 0xFFu));
    const __half2 f2 = __half2half2(fh), nb2 = __half2half2(__hmul(__float2half_rn(-1024.0f), fh));
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t n0 = (w[2 * c] >> (4 * sl)) & 0x0F0F0F0Fu, n1 = (w[2 * c + 1] >> (4 * sl)) & 0x0F0F0F0Fu;
      *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + c)) =
          make_uint4(x_hfma2(prmt(n0, 0x64646464u, 0x4140u), f2, nb2), x_hfma2(prmt(n0, 0x64646464u, 0x4342u), f2, nb2),
                     x_hfma2(prmt(n1, 0x64646464u, 0x4140u), f2, nb2), x_hfma2(prmt(n1, 0x64646464u, 0x4342u), f2, nb2));
    }
  }
  if (kb == 0) *dw = sigma;
  const float fm = -16.0f * h2f(hdr.x >> 16) / sigma, fs = 128.0f * ratio;
  *reinterpret_cast<__half2*>(ta + 4 * kb) = __floats2half2_rn(fm * (float)(mn & 0xFFu), fm * (float)(mn >> 8));
  *reinterpret_cast<__half2*>(ta + 128 + 4 * kb) = __floats2half2_rn(fs * (float)(sc & 0xFFu), fs * (float)(sc >> 8));
}

// IQ3_S records (layout: gsq_repack.cu). Warp w: record w / 2, half w % 2 of the superblock; thread i plays lane
// (i % 8) * 4 + i / 8 of the record, so that eight threads store to eight different rows of a group.
template <int HF>
__device__ __forceinline__ void x_iq3s_packed(const uint8_t* p, uint8_t* out, const uint8_t* grid, int rec, int thread) {
  const int gq = thread & 7, t = thread >> 3, lane = 4 * gq + t;
  const uint32_t lane_off = (uint32_t)(thread & (GRID_REP - 1)) << 3;
  uint32_t idx[5];
  if (HF == 0) {
    const uint4 ia = *reinterpret_cast<const uint4*>(p + 16 * lane);
    idx[0] = ia.x; idx[1] = ia.y; idx[2] = ia.z; idx[3] = ia.w;
    idx[4] = *reinterpret_cast<const uint32_t*>(p + 512 + 16 * lane);
  } else {
    const uint4 ib = *reinterpret_cast<const uint4*>(p + 512 + 16 * lane);
    idx[0] = ib.x; idx[1] = ib.y; idx[2] = ib.z; idx[3] = ib.w;
    idx[4] = *reinterpret_cast<const uint32_t*>(p + 1024 + 4 * lane);
  }
  const uint2 sgw2 = *reinterpret_cast<const uint2*>(p + 1152 + 16 * lane + 8 * HF);
  const uint2 sc = *reinterpret_cast<const uint2*>(p + 1664 + 8 * gq);
#pragma unroll
  for (int sh = 0; sh < 4; ++sh) {               // slice within the half
    const int s = 4 * HF + sh;
    const uint32_t sgw = sh < 2 ? sgw2.x : sgw2.y;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t wv[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int f = 4 * sh + 2 * h + e;        // field within the half
        const int bit = 9 * f + 16 * HF, word = bit >> 5, off = bit & 31;
        // index << 5: times the 32 bytes of an entry's replicas
        uint32_t v;
        if (off + 9 <= 32) v = off >= 5 ? idx[word] >> (off >= 5 ? off - 5 : 0) : idx[word] << (off < 5 ? 5 - off : 0);
        else v = __funnelshift_r(idx[word], idx[word + 1], off - 5);
        const uint2 gp = *reinterpret_cast<const uint2*>(grid + ((v & 0x3FE0u) | lane_off));
        const int fl = f & 7, sft = 16 * (fl >> 2) + (fl & 3) - 2;
        const uint32_t sgs = sft >= 0 ? sgw >> (sft >= 0 ? sft : 0) : sgw << (sft < 0 ? -sft : 0);
        wv[e] = prmt(gp.x, gp.y, (sgs & 0x4444u) | 0x3210u);
      }
      const Sub sub(1 + 2 * (int)(((h ? sc.y : sc.x) >> (4 * s)) & 15u));
      *reinterpret_cast<uint4*>(out + out_at(2 * HF + (sh >> 1), 0, 1, 16 * rec + gq + 8 * h, 4 * (sh & 1) + t)) = scale8(wv[0], wv[1], sub);
    }
  }
}

// Q6_K records: warp w: record w / 2, row g + 8 (w % 2) of lane 4 g + t
__device__ __forceinline__ void x_q6k_packed(const uint8_t* p, uint8_t* out, int rec, int h, int lane, float* dw) {
  const int g = lane >> 2, t = lane & 3, r = 16 * rec + g + 8 * h;
  const uint4 la = *reinterpret_cast<const uint4*>(p + 64 * lane + 32 * h), lb = *reinterpret_cast<const uint4*>(p + 64 * lane + 32 * h + 16);
  const uint4 qh = *reinterpret_cast<const uint4*>(p + 2048 + 32 * lane + 16 * h);
  const uint4 sc = *reinterpret_cast<const uint4*>(p + 3072 + 32 * g + 16 * h);
  const uint32_t ql[8] = {la.x, la.y, la.z, la.w, lb.x, lb.y, lb.z, lb.w}, hi2[4] = {qh.x, qh.y, qh.z, qh.w}, sw[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
  for (int n = 0; n < 2; ++n) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
      for (int is = 0; is < 2; ++is) {
        const uint32_t lw = ql[4 * n + 2 * (q & 1) + is], hw = hi2[2 * n + is];
        const uint32_t v = ((lw >> (q & 2 ? 4 : 0)) & 0x0F0F0F0Fu) | (((hw >> (2 * q)) & 0x03030303u) << 4);
        const int G = 8 * n + 2 * q + is;
        const int scv = (int)(int8_t)(sw[G >> 2] >> (8 * (G & 3)));
        uint2 hi, lo;
        scale4_pair(v + 0x60606060u, __half2half2(__int2half_rn(scv)), hi, lo);   // q - 32 + 128, no carries
        *reinterpret_cast<uint2*>(out + out_at(G >> 2, 0, 2, r, 2 * (G & 3) + (t >> 1)) + 8 * (t & 1)) = hi;
        *reinterpret_cast<uint2*>(out + out_at(G >> 2, 1, 2, r, 2 * (G & 3) + (t >> 1)) + 8 * (t & 1)) = lo;
      }
    }
  }
  if (t == 0) *dw = h2f(*reinterpret_cast<const uint16_t*>(p + 3328 + 4 * g + 2 * h));
}

// IQ3_S and Q6_K in GGUF order (layers that are not repacked)
__device__ __forceinline__ void x_iq3s(const uint8_t* s, uint8_t* out, const uint8_t* grid, int r, int kb, float* dw) {
#pragma unroll
  for (int sl = 0; sl < 2; ++sl) {
    const int p = 2 * kb + sl;
    const uint32_t qh = s[66 + p];
    const Sub sub(1 + 2 * (int)((s[106 + kb] >> (4 * sl)) & 15));
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint32_t sg = s[74 + 4 * p + c];
      uint32_t v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t i = (uint32_t)s[2 + 8 * p + 2 * c + e] | (((qh >> (2 * c + e)) & 1u) << 8);
        const uint2 gp = *reinterpret_cast<const uint2*>(grid + i * (8 * GRID_REP) + 8 * (threadIdx.x & (GRID_REP - 1)));
        const uint32_t b = sg >> (4 * e);
        v[e] = prmt(gp.x, gp.y, 0x3210u | ((b & 1u) << 2) | ((b & 2u) << 5) | ((b & 4u) << 8) | ((b & 8u) << 11));
      }
      *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + c)) = scale8(v[0], v[1], sub);
    }
  }
  if (kb == 0) *dw = h2f(*reinterpret_cast<const uint16_t*>(s));
}
__device__ __forceinline__ void x_q6k(const uint8_t* s, uint8_t* out, int r, int kb, float* dw) {
  const int n = kb >> 1;
#pragma unroll
  for (int c = 0; c < 8; ++c) {                  // chunk of 8 values: values 64 kb + 8 c ..
    const int qt = 2 * (kb & 1) + (c >> 2), l0 = 8 * (c & 3);
    const int scv = (int)(int8_t)s[192 + 8 * n + 2 * qt + (l0 >> 4)];
    uint2 hi[2], lo[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int l = l0 + 4 * e;
      const uint32_t lw = (uint32_t)*reinterpret_cast<const uint16_t*>(s + 64 * n + 32 * (qt & 1) + l) |
                          ((uint32_t)*reinterpret_cast<const uint16_t*>(s + 64 * n + 32 * (qt & 1) + l + 2) << 16);
      const uint32_t hw = (uint32_t)*reinterpret_cast<const uint16_t*>(s + 128 + 32 * n + l) |
                          ((uint32_t)*reinterpret_cast<const uint16_t*>(s + 128 + 32 * n + l + 2) << 16);
      const uint32_t v = ((qt & 2 ? lw >> 4 : lw) & 0x0F0F0F0Fu) | (((hw >> (2 * qt)) & 0x03030303u) << 4);
      scale4_pair(v + 0x60606060u, __half2half2(__int2half_rn(scv)), hi[e], lo[e]);
    }
    *reinterpret_cast<uint4*>(out + out_at(kb, 0, 2, r, c)) = make_uint4(hi[0].x, hi[0].y, hi[1].x, hi[1].y);
    *reinterpret_cast<uint4*>(out + out_at(kb, 1, 2, r, c)) = make_uint4(lo[0].x, lo[0].y, lo[1].x, lo[1].y);
  }
  if (kb == 0) *dw = h2f(*reinterpret_cast<const uint16_t*>(s + 208));
}

// The low-bit types: decoded by the codec they share with the dp4a kernel and the row dequantiser. Factor per row and
// superblock: the truncating integer divisions of the reference's small-row kernels (its many-row kernels scale in
// floating point, as here) become the exact fractions d / 8, d / 4. (The truncation is 1e-5 to 5e-5 of a result's norm, so
// a type's results change by that where its rows pass from the one kernel to the other, and are nearer to 64 bits above.)
template <int F1>
__device__ __forceinline__ void x_f1(const uint8_t* s, uint8_t* out, int r, int kb, float* dw, float* dm, uint8_t* ta) {
#pragma unroll
  for (int sl = 0; sl < 2; ++sl) {
    Raw<F1> raw;
    raw.template fetch<true>(s, 2 * kb + sl);
    Slice<F1> v;
    v.decode(raw, 2 * kb + sl);
    int f0, f1;
    if (F1 == F1_IQ2XXS || F1 == F1_IQ3XXS) { f0 = f1 = 2 * v.p0 + 1; }
    else if (F1 == F1_IQ2XS || F1 == F1_IQ2S) { f0 = 2 * v.p0 + 1; f1 = 2 * v.p1 + 1; }
    else { f0 = v.p0; f1 = v.p1; }
    if constexpr (F1 == F1_Q2K) {
      // 0..3 under the high byte 0x64: (1024 + value) * sc - 1024 * sc, exact
      const __half h0 = __int2half_rn(f0), h1 = __int2half_rn(f1);
      const __half2 m0 = __half2half2(h0), m1 = __half2half2(h1);
      const __half2 n0 = __half2half2(__hmul(__float2half_rn(-1024.0f), h0)), n1 = __half2half2(__hmul(__float2half_rn(-1024.0f), h1));
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const __half2 f = c < 2 ? m0 : m1, nb = c < 2 ? n0 : n1;
        const uint32_t a = (uint32_t)v.wv[2 * c], b = (uint32_t)v.wv[2 * c + 1];
        *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + c)) =
            make_uint4(x_hfma2(prmt(a, 0x64646464u, 0x4140u), f, nb), x_hfma2(prmt(a, 0x64646464u, 0x4342u), f, nb),
                       x_hfma2(prmt(b, 0x64646464u, 0x4140u), f, nb), x_hfma2(prmt(b, 0x64646464u, 0x4342u), f, nb));
      }
      // the minimums of the two 16-value groups, against the sums of their quants; -dmin scales them
      *reinterpret_cast<__half2*>(ta + (kb >> 1) * 128 + (kb & 1) * 8 + 4 * sl) = __halves2half2(__int2half_rn(v.p2), __int2half_rn(v.p3));
      if (kb == 0 && sl == 0) {
        *dw = v.d;
        *dm = -v.dmin;
      }
    } else {
      const Sub s0(f0), s1(f1);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t a = (uint32_t)v.wv[2 * c], b = (uint32_t)v.wv[2 * c + 1];
        if (F1 == F1_IQ1M) {
          // codebook value + 1 in 0..2, delta +-1/8: 8 (value) +- 1, biased by 128
          const uint32_t bias = ((v.p2 >> c) & 1) ? 0x77777777u : 0x79797979u;
          a = (a << 3) + bias;
          b = (b << 3) + bias;
        } else {
          a ^= 0x80808080u;
          b ^= 0x80808080u;
        }
        *reinterpret_cast<uint4*>(out + out_at(kb, 0, 1, r, 4 * sl + c)) = scale8(a, b, c < 2 ? s0 : s1);
      }
      if (kb == 0 && sl == 0) *dw = v.d * (F1 == F1_IQ3XXS ? 0.25f : 0.125f);
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(XTHREADS) expand_kernel(const ExpandArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  using T = typename Unit<x_unit(KIND)>::T;
  constexpr int PER = x_segment(KIND) / x_unit(KIND), UNITS = x_segments(KIND) * PER, NLD = (UNITS + XTHREADS - 1) / XTHREADS;
  constexpr int AP = a_planes(KIND), TP = t_planes(KIND);
  uint8_t* const out = smem;
  uint8_t* const grid = smem + x_out(KIND);
  uint8_t* const raw0 = grid + x_table(KIND);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (x_table(KIND)) {
    for (int i = tid; i < 512; i += XTHREADS) {
      const uint32_t gv = g_x_iq3s_grid[i];
      const uint32_t pos = gv ^ 0x80808080u, neg = (~gv + 0x01010101u) ^ 0x80808080u;   // no codebook byte is zero
#pragma unroll
      for (int q = 0; q < GRID_REP / 2; ++q) reinterpret_cast<uint4*>(grid + i * 8 * GRID_REP)[q] = make_uint4(pos, neg, pos, neg);
    }
  }
  // items: superblock fastest, so that a CTA's neighbours read neighbouring bytes of the same rows
  T reg[NLD];
  auto load = [&](int item) {
    const int ht = item / g.nsb, sb = item - ht * g.nsb;
#pragma unroll
    for (int i = 0; i < NLD; ++i) {
      const int u = tid + i * XTHREADS, seg = u / PER, c = u - seg * PER;
      const int row = ht * XROWS + (x_packed(KIND) ? 16 : 1) * seg;
      if (u < UNITS && row < g.nrows)
        reg[i] = __ldg(reinterpret_cast<const T*>(g.w + (int64_t)row * g.row_bytes + (int64_t)sb * x_segment(KIND)) + c);
    }
  };
  auto stash = [&](uint8_t* raw) {
#pragma unroll
    for (int i = 0; i < NLD; ++i) {
      const int u = tid + i * XTHREADS, seg = u / PER, c = u - seg * PER;
      if (u < UNITS) *reinterpret_cast<T*>(raw + seg * x_stride(KIND) + c * (int)sizeof(T)) = reg[i];
    }
  };
#pragma unroll
  for (int i = 0; i < NLD; ++i) reg[i] = T{};
  int item = blockIdx.x;
  if (item < g.n_items) load(item);
  // the weights may be read before the previous kernel has finished; the operand buffer may not be written
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // Only now may the next kernel start: where that is the one that quantises the activations (gsq_planes.cu), it takes it that
  // whatever ran before this kernel has finished, and runs beside this one.
  asm volatile("griddepcontrol.launch_dependents;");
  for (int n = 0; item < g.n_items; ++n) {
    uint8_t* const raw = raw0 + (n & 1) * x_raw(KIND);
    stash(raw);
    const int next = item + gridDim.x;
    if (next < g.n_items) load(next);
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the last item has left the out buffer
    __syncthreads();
    const int ht = item / g.nsb, sb = item - ht * g.nsb, rt = ht >> 1, half = ht & 1;
    float* const dw = g.dw + ((int64_t)rt * g.nsb + sb) * TR + half * XROWS;
    float* const dm = KIND == K_Q2K ? g.dm + (dw - g.dw) : nullptr;
    uint8_t* const ta = TP ? g.ta + ((int64_t)rt * g.nsb + sb) * 4096 + half * (XROWS / 8 * 256) : nullptr;
    if constexpr (x_packed(KIND)) {
      const int rec = warp >> 1, hf = warp & 1;
      if (ht * XROWS + 16 * rec < g.nrows) {
        const uint8_t* p = raw + rec * x_stride(KIND);
        if (KIND == K_IQ3S_PACKED) {
          if (hf == 0) x_iq3s_packed<0>(p, out, grid, rec, lane);
          else x_iq3s_packed<1>(p, out, grid, rec, lane);
          if (hf == 0 && lane < 16) dw[16 * rec + lane] = h2f(*reinterpret_cast<const uint16_t*>(p + 1728 + 4 * (lane & 7) + 2 * (lane >> 3)));
        } else {
          x_q6k_packed(p, out, rec, hf, lane, dw + 16 * rec + (lane >> 2) + 8 * hf);
        }
      } else {
        // 16 rows past the last one: this warp's half of their tile as zeros
#pragma unroll
        for (int kb = 2 * hf; kb < 2 * hf + 2; ++kb)
          for (int pln = 0; pln < AP; ++pln)
            for (int i = lane; i < 128; i += 32) *reinterpret_cast<uint4*>(out + out_at(kb, pln, AP, 16 * rec + (i >> 3), i & 7)) = make_uint4(0, 0, 0, 0);
        if (hf == 0 && lane < 16) dw[16 * rec + lane] = 0.0f;
      }
    } else {
      const int r = tid & 63, kb = tid >> 6;
      const uint8_t* s = raw + r * x_stride(KIND);
      uint8_t* const tar = TP ? ta + (r >> 3) * 256 + (r & 7) * 16 : nullptr;
      if (ht * XROWS + r < g.nrows) {
        if (KIND == K_Q4K) x_q4k(s, out, r, kb, dw + r, tar);
        else if (KIND == K_IQ4XS) x_iq4xs(s, out, r, kb, dw + r);
        else if (KIND == K_IQ3S) x_iq3s(s, out, grid, r, kb, dw + r);
        else if (KIND == K_Q6K) x_q6k(s, out, r, kb, dw + r);
        else x_f1<KIND == K_Q2K ? F1_Q2K : KIND == K_IQ2XXS ? F1_IQ2XXS : KIND == K_IQ2XS ? F1_IQ2XS : KIND == K_IQ2S ? F1_IQ2S
                  : KIND == K_IQ3XXS ? F1_IQ3XXS : F1_IQ1M>(s, out, r, kb, dw + r, dm + r, tar);
      } else {
        for (int pln = 0; pln < AP; ++pln)
#pragma unroll
          for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(out + out_at(kb, pln, AP, r, c)) = make_uint4(0, 0, 0, 0);
        if (kb == 0) dw[r] = 0.0f;
        if (KIND == K_Q2K && kb == 0) dm[r] = 0.0f;
        if (TP && kb < 2) *reinterpret_cast<uint4*>(tar + kb * 128) = make_uint4(0, 0, 0, 0);
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
#pragma unroll
      for (int i = 0; i < 4 * AP; ++i) {
        uint8_t* dst = g.a + ((int64_t)rt * (4 * g.nsb) + 4 * sb) * (AP * A_TILE) + (int64_t)i * A_TILE + half * (A_TILE / 2);
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(tc::saddr(out + i * (A_TILE / 2))),
                     "r"(A_TILE / 2)
                     : "memory");
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    item = next;
  }
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

template <int KIND>
static int launch_expand(const ExpandArgs& g, int sm_count, cudaStream_t st) {
  constexpr int smem = x_smem(KIND);
  static_assert(smem <= 227 * 1024, "shared memory budget");
  static std::atomic<int> per_sm[64];
  int dev = 0;
  GSQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return GSQ_ERR_UNSUPPORTED;
  if (!per_sm[dev]) {
    GSQ_CUDA_TRY(cudaFuncSetAttribute(expand_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int n = 0;
    GSQ_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, expand_kernel<KIND>, XTHREADS, smem));
    if (n < 1) return GSQ_ERR_UNSUPPORTED;
    per_sm[dev] = n;
  }
  cudaLaunchConfig_t cfg = {};
  const int most = per_sm[dev] * sm_count;
  cfg.gridDim = dim3((unsigned)(g.n_items < most ? g.n_items : most));
  cfg.blockDim = dim3(XTHREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, expand_kernel<KIND>, g));
  return GSQ_OK;
}

// rows [0, rows) of w (rows of this call) -> operand tiles of ceil(rows / 256) pairs of row tiles
int expand_host(const Plan& p, const uint8_t* w, int64_t row_bytes, int64_t rows, uint8_t* scratch, int sm_count, cudaStream_t st) {
  ExpandArgs g;
  g.w = w;
  g.row_bytes = row_bytes;
  g.nrows = (int)rows;
  g.nsb = p.nsb;
  g.n_items = (int)((rows + 255) / 256 * 4) * p.nsb;
  g.a = scratch + p.a;
  g.dw = reinterpret_cast<float*>(scratch + p.dw);
  g.dm = reinterpret_cast<float*>(scratch + p.dm);
  g.ta = scratch + p.ta;
  switch (p.kind) {
    case K_Q4K: return launch_expand<K_Q4K>(g, sm_count, st);
    case K_IQ4XS: return launch_expand<K_IQ4XS>(g, sm_count, st);
    case K_IQ3S_PACKED: return launch_expand<K_IQ3S_PACKED>(g, sm_count, st);
    case K_Q6K_PACKED: return launch_expand<K_Q6K_PACKED>(g, sm_count, st);
    case K_IQ3S: return launch_expand<K_IQ3S>(g, sm_count, st);
    case K_Q6K: return launch_expand<K_Q6K>(g, sm_count, st);
    case K_Q2K: return launch_expand<K_Q2K>(g, sm_count, st);
    case K_IQ2XXS: return launch_expand<K_IQ2XXS>(g, sm_count, st);
    case K_IQ2XS: return launch_expand<K_IQ2XS>(g, sm_count, st);
    case K_IQ2S: return launch_expand<K_IQ2S>(g, sm_count, st);
    case K_IQ3XXS: return launch_expand<K_IQ3XXS>(g, sm_count, st);
    case K_IQ1M: return launch_expand<K_IQ1M>(g, sm_count, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}

}  // namespace pl
}  // namespace gsq
