// Product of a few tens to 256 activation rows with exact integer slice sums (sm_100a: tcgen05 kind::i8), weights decoded
// in the kernel: repacked IQ3_S, IQ4_XS and Q4_K. The arithmetic is that of the reference's many-row kernels
// (csrc/lcpp/ggml/src/ggml-cuda/mmq.cuh:961-1385): int32 dot products of 32-value slices, scaled by d * sub-scale of the
// row and d of the token in fp32.
//
// What bounds it: at these row counts reading the weights takes 6 us for 17408 x 5120; decoding them (about 2 instructions
// per value) and scaling the sums (3 per row, token and slice) keep the issue slots and the logic pipe of all SMs busy for
// several times that, so the work is spread evenly and everything else kept off those pipes:
//   * The units of work are (128-row tile, superblock); every CTA takes the same number of consecutive ones (+-1), cut
//     anywhere inside a tile. A tile finished by one CTA is stored directly; parts of a tile go to scratch as fp32 and a
//     second kernel adds them in order.
//   * 8 producer warps decode a superblock of 128 rows ONCE for all tokens into an int8 operand tile; one warp issues one
//     128 x nt x 32 instruction per slice; the consumer warps scale the sums into registers; one thread copies the
//     activation units. All hand-offs are mbarriers.
//   * The IQ3_S codebook is in shared memory 32 times, once per bank: a look-up never conflicts. A codebook byte g is odd,
//     so -g is g ^ 0xFE: one instruction gives the negated group that the sign selectors pick from.
//   * Q4_K's minimum term is one more instruction per superblock (kind::f16: 6-bit minimums times half(sum x), exact),
//     scaled once per superblock instead of once per slice.
#pragma once
#include <cuda_fp16.h>

#include "gsq_common.cuh"
#include "gsq_quant.cuh"
#include "gsq_tables.h"
#include "gsq_tc.cuh"

namespace gsq {
namespace g5 {

using namespace tc;

enum { G5_IQ3S = 0, G5_IQ4XS = 1, G5_Q4K = 2 };

constexpr int TR = 128;
constexpr int PROD_WARPS = 8, PROD_THREADS = 256;
constexpr int CONS_WARP0 = 8, CONS_WARPS = 16;      // four per tensor-memory lane quarter, a quarter of the tokens each
constexpr int MMA_WARP = 24, COPY_WARP = 25, THREADS = 896;
// registers: 896 threads start with 72 each; the warpgroup of the MMA and copy warps gives up 48, everyone else takes 8
constexpr int IDLE_REGS = 24, WORK_REGS = 80;
constexpr int SL_A = TR * 32;                       // one slice of the weight tile
constexpr int A_STAGES = 2;                         // (the minimum term's two tensor-memory buffers rely on 2)
constexpr int RAW_STAGES = 2;
constexpr int MAX_B = 4;
constexpr int TMEM_COLS = 512;
constexpr int MAX_NT = 128;

__host__ __device__ constexpr int raw_row(int kind) { return kind == G5_IQ4XS ? 136 : 144; }
__host__ __device__ constexpr int raw_bytes(int kind) { return kind == G5_IQ3S ? 0 : TR * raw_row(kind); }
__host__ __device__ constexpr int table_bytes(int kind) { return kind == G5_IQ3S ? 512 * 128 : 0; }
// weight stage: 8 slices, d * sub-scale per slice and row; Q4_K: dmin per row, the 6-bit minimums as a 16-column fp16 operand
__host__ __device__ constexpr int a_stage(int kind) { return 8 * SL_A + 8 * TR * 4 + (kind == G5_Q4K ? TR * 4 + TR * 32 : 0); }
// activation unit of one superblock and nt tokens: 8 slices of int8 operand, d per slice and token; Q4_K: half(sum x) operand
__host__ __device__ constexpr int unit_bytes(bool ds, int nt) { return nt * (256 + 32 + (ds ? 32 : 0)); }

struct Args {
  const uint8_t* w;
  int64_t row_bytes;
  int nrows, nsb, n_rt, n_units;
  const uint8_t* xb;       // [token block][superblock][unit]
  int nt, m, b_stages;
  void* y;
  int y_dtype;
  int64_t ldy;
  float* part;             // [2 * CTA + which][nt][128]
};

struct Smem {
  int table, raw, a, b, total;
};
__host__ __device__ inline Smem smem_map(int kind, int nt, int b_stages) {
  Smem s;
  s.table = 1024;
  s.raw = s.table + table_bytes(kind);
  s.a = s.raw + RAW_STAGES * raw_bytes(kind);
  s.b = s.a + A_STAGES * a_stage(kind);
  s.total = s.b + b_stages * unit_bytes(kind == G5_Q4K, nt);
  return s;
}

static __device__ int g_error = 0;   // (one per translation unit: one per weight type)
static __device__ const uint32_t g_grid[512] = GSQ_IQ3S_GRID_INIT;
static __constant__ __align__(16) int8_t c_iq4nl5[16] = GSQ_IQ4NL_VALUES_INIT;

struct Ring {
  uint32_t i, ph;
  __device__ __forceinline__ void next(uint32_t n) {
    if (++i == n) { i = 0; ph ^= 1u; }
  }
};

__device__ __forceinline__ bool try_bar(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// bounded: about a second after the first failed try, or when another thread of the CTA has given up.
// `ns`: pause between tries -- a waiting warp should not spend the issue slots of the working ones on polls
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag, uint32_t ns) {
  if (try_bar(bar, parity)) return true;
  const long long t0 = clock64();
  for (int spin = 1; spin < (1 << 28); ++spin) {
    if (ns) __nanosleep(ns);
    if (try_bar(bar, parity)) return true;
    if ((spin & 15) == 0 && (*abort_flag || clock64() - t0 > 2000000000ll)) break;
  }
  if (!*abort_flag) {
    *abort_flag = 1;
    atomicExch(&g_error, 1);
  }
  return false;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
  return r != 0;
}
// 16-byte piece c16 of row r inside one slice of a K-major int8 tile
__device__ __forceinline__ int core_off(int r, int c16) { return (r >> 3) * 256 + c16 * 128 + (r & 7) * 16; }

// ---------------------------------------------------------------------------------------------
// Producers.

// IQ3_S: one record (16 rows of a superblock; layout: gsq_repack.cu) per warp, straight from global memory into
// registers, the next one's loads in flight while one is decoded. Thread i plays lane (i % 8) * 4 + i / 8, so that the
// threads of a half warp store to eight rows' 16-byte pieces.
struct Rec3 {
  uint4 ia, ib, sg;
  uint2 sc;
  uint32_t i8, dd;
  __device__ __forceinline__ void load(const uint8_t* p, int lane, int gq) {
    ia = ldg_stream_v4(p + 16 * lane);
    ib = ldg_stream_v4(p + 512 + 16 * lane);
    i8 = ldg_stream_u32(p + 1024 + 4 * lane);
    sg = ldg_stream_v4(p + 1152 + 16 * lane);
    sc = ldg_stream_v2(p + 1664 + 8 * gq);
    dd = ldg_stream_u32(p + 1728 + 4 * gq);
  }
};
__device__ __forceinline__ void decode_iq3s(const Rec3& q, uint8_t* a, float* f, const uint8_t* table, int rec, int gq, int t, int thread) {
  const uint32_t idx[9] = {q.ia.x, q.ia.y, q.ia.z, q.ia.w, q.ib.x, q.ib.y, q.ib.z, q.ib.w, q.i8};
  const uint32_t sgw[4] = {q.sg.x, q.sg.y, q.sg.z, q.sg.w};
  const uint8_t* tab = table + 4 * thread;
#pragma unroll
  for (int s = 0; s < 8; ++s) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t wv[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int fld = 4 * s + 2 * h + e, bit = 9 * fld, word = bit >> 5, off = bit & 31;
        // index * 128: bytes of an entry's 32 copies
        uint32_t v;
        if (off + 9 <= 32) v = off >= 7 ? idx[word] >> (off >= 7 ? off - 7 : 0) : idx[word] << (off < 7 ? 7 - off : 0);
        else v = __funnelshift_r(idx[word], idx[word + 1], off - 7);
        const uint32_t g = *reinterpret_cast<const uint32_t*>(tab + (v & 0xFF80u));
        const int fl = fld & 7, sft = 16 * (fl >> 2) + (fl & 3) - 2;
        const uint32_t w = sgw[fld >> 3];
        const uint32_t sel = sft >= 0 ? w >> (sft >= 0 ? sft : 0) : w << (sft < 0 ? -sft : 0);
        wv[e] = prmt(g, g ^ 0xFEFEFEFEu, (sel & 0x4444u) | 0x3210u);
      }
      *reinterpret_cast<uint2*>(a + s * SL_A + core_off(16 * rec + gq + 8 * h, t >> 1) + 8 * (t & 1)) = make_uint2(wv[0], wv[1]);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float d = h2f(q.dd >> (16 * h));
    const uint32_t scw = (h ? q.sc.y : q.sc.x) >> (8 * t);     // slices 2 t, 2 t + 1
    f[(2 * t) * TR + 16 * rec + gq + 8 * h] = d * (float)(1 + 2 * (int)(scw & 15u));
    f[(2 * t + 1) * TR + 16 * rec + gq + 8 * h] = d * (float)(1 + 2 * (int)((scw >> 4) & 15u));
  }
}

__device__ __forceinline__ void iq4_lookup(uint32_t v, const uint32_t (&tb)[4], uint32_t& lo, uint32_t& hi) {
  // (a byte permute reads the low 16 bits of its selector, so the upper four nibbles' selectors are one shift away)
  const uint32_t s01 = v & 0x77777777u, s23 = s01 >> 16;
  const uint32_t pick01 = ((v >> 1) & 0x44444444u) | 0x32103210u, pick23 = pick01 >> 16;
  const uint32_t r01 = prmt(prmt(tb[0], tb[1], s01), prmt(tb[2], tb[3], s01), pick01);
  const uint32_t r23 = prmt(prmt(tb[0], tb[1], s23), prmt(tb[2], tb[3], s23), pick23);
  lo = prmt(r01, r23, 0x6420u);
  hi = prmt(r01, r23, 0x7531u);
}
// GGUF-order types: thread = row r, half `hf` of the superblock (4 slices), raw blocks in shared memory
__device__ __forceinline__ void decode_iq4xs(const uint8_t* b, uint8_t* a, float* f, int r, int hf) {
  const uint32_t* tw = reinterpret_cast<const uint32_t*>(c_iq4nl5);
  const uint32_t tb[4] = {tw[0], tw[1], tw[2], tw[3]};
  const uint2 hdr = *reinterpret_cast<const uint2*>(b);
  const float d = h2f(hdr.x);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int s = 4 * hf + i;
    const uint2 qa = *reinterpret_cast<const uint2*>(b + 8 + 16 * s), qb = *reinterpret_cast<const uint2*>(b + 16 + 16 * s);
    const uint32_t v[4] = {qa.x, qa.y, qb.x, qb.y};
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) iq4_lookup(v[e], tb, lo[e], hi[e]);
    *reinterpret_cast<uint4*>(a + s * SL_A + core_off(r, 0)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    *reinterpret_cast<uint4*>(a + s * SL_A + core_off(r, 1)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    f[s * TR + r] = d * (float)((int)(((hdr.y >> (4 * s)) & 0xFu) | (((hdr.x >> (16 + 2 * s)) & 3u) << 4)) - 32);
  }
}
__device__ __forceinline__ void decode_q4k(const uint8_t* b, uint8_t* a, float* f, float* fmin, uint8_t* amin, int r, int hf) {
  const uint4 hdr = *reinterpret_cast<const uint4*>(b);
  const float d = h2f(hdr.x);
  __half2 mins[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int jj = 2 * hf + i;
    const uint4 va = *reinterpret_cast<const uint4*>(b + 16 + 32 * jj), vb = *reinterpret_cast<const uint4*>(b + 32 + 32 * jj);
    const uint32_t w[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
#pragma unroll
    for (int hi = 0; hi < 2; ++hi) {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint4 o;
        o.x = (w[4 * c] >> (4 * hi)) & 0x0F0F0F0Fu;
        o.y = (w[4 * c + 1] >> (4 * hi)) & 0x0F0F0F0Fu;
        o.z = (w[4 * c + 2] >> (4 * hi)) & 0x0F0F0F0Fu;
        o.w = (w[4 * c + 3] >> (4 * hi)) & 0x0F0F0F0Fu;
        *reinterpret_cast<uint4*>(a + (2 * jj + hi) * SL_A + core_off(r, c)) = o;
      }
    }
    const uint32_t selh = (jj & 1) ? 0x4432u : 0x4410u;
    const uint32_t A = prmt(hdr.y, 0u, selh), B = prmt(hdr.z, 0u, selh), C = prmt(hdr.w, 0u, selh);
    const uint32_t sc = jj < 2 ? (A & 0x3F3Fu) : ((C & 0x0F0Fu) | ((A & 0xC0C0u) >> 2));
    const uint32_t mn = jj < 2 ? (B & 0x3F3Fu) : (((C >> 4) & 0x0F0Fu) | ((B & 0xC0C0u) >> 2));
    f[(2 * jj) * TR + r] = d * (float)(sc & 0xFFu);
    f[(2 * jj + 1) * TR + r] = d * (float)(sc >> 8);
    mins[i] = __floats2half2_rn((float)(mn & 0xFFu), (float)(mn >> 8));
  }
  // row r of the 16-column operand: minimums of slices 0..7, then 8 columns of zeros
  uint8_t* dst = amin + (r >> 3) * 256 + (r & 7) * 16;
  *reinterpret_cast<uint2*>(dst + 8 * hf) = *reinterpret_cast<const uint2*>(mins);
  *reinterpret_cast<uint2*>(dst + 128 + 8 * hf) = make_uint2(0u, 0u);
  if (hf == 0) fmin[r] = -h2f(hdr.x >> 16);
}

// a walk over consecutive units: superblock fastest, then row tile, then token block (one division, at the start)
struct Unit {
  int sb, rt, tb;
  __device__ __forceinline__ Unit(const Args& g, int u) {
    const int tile = u / g.nsb;
    sb = u - tile * g.nsb;
    tb = tile / g.n_rt;
    rt = tile - tb * g.n_rt;
  }
  __device__ __forceinline__ void next(const Args& g) {
    if (++sb == g.nsb) {
      sb = 0;
      if (++rt == g.n_rt) { rt = 0; ++tb; }
    }
  }
};

template <int KIND>
__device__ __forceinline__ void fetch_raw(const Args& g, const Unit& at, uint8_t* raw, int ptid) {
  const int rt = at.rt, sb = at.sb;
  const uint32_t dst = saddr(raw);
  constexpr int PER = KIND == G5_IQ4XS ? 17 : 9, U = KIND == G5_IQ4XS ? 8 : 16;
  for (int i = ptid; i < TR * PER; i += PROD_THREADS) {
    const int r = i / PER, c = i - r * PER;
    const int row = min(rt * TR + r, g.nrows - 1);   // rows past the last one repeat it (their results are not stored)
    const uint8_t* src = g.w + (int64_t)row * g.row_bytes + (int64_t)sb * raw_row(KIND) + c * U;
    if (KIND == G5_IQ4XS) cp_async8(dst + r * raw_row(KIND) + c * U, src);
    else cp_async16(dst + r * raw_row(KIND) + c * U, src);
  }
}

// ---------------------------------------------------------------------------------------------
// Consumers.

// Tensor-memory loads without a memory clobber: what they read is not memory to the compiler, and the shared-memory loads
// of the token scales may move across them (the wait's data dependency is the pin below it).
__device__ __forceinline__ void ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
}
__device__ __forceinline__ void ld_wait(uint32_t (&v)[8]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]));
}

// N columns (4 or 8) of one slice: acc += (C * f) * d. C * f is formed as fma(bits(1.5 * 2^23 + C), f, -1.5 * 2^23 * f):
// f has at most 17 significant bits, so the subtrahend is exact and the result the correctly rounded product.
template <int N>
__device__ __forceinline__ void scale(const uint32_t (&c)[8], float2 f2, float2 nf2, const float* bd, float2* acc) {
#pragma unroll
  for (int j = 0; j < N / 4; ++j) {
    const float4 d = *reinterpret_cast<const float4*>(bd + 4 * j);
    const float2 t0 = __ffma2_rn(make_float2(biased_float(c[4 * j]), biased_float(c[4 * j + 1])), f2, nf2);
    const float2 t1 = __ffma2_rn(make_float2(biased_float(c[4 * j + 2]), biased_float(c[4 * j + 3])), f2, nf2);
    acc[2 * j].x = fmaf(t0.x, d.x, acc[2 * j].x);
    acc[2 * j].y = fmaf(t0.y, d.y, acc[2 * j].y);
    acc[2 * j + 1].x = fmaf(t1.x, d.z, acc[2 * j + 1].x);
    acc[2 * j + 1].y = fmaf(t1.y, d.w, acc[2 * j + 1].y);
  }
}

template <typename T, int CP>
__device__ __forceinline__ void store_cols(T* y, int64_t ld, const float2 (&acc)[CP / 2], int n) {
#pragma unroll
  for (int i = 0; i < CP / 2; ++i) {
    if (2 * i < n) store_out<T>(y + (2 * i) * ld, acc[i].x);
    if (2 * i + 1 < n) store_out<T>(y + (2 * i + 1) * ld, acc[i].y);
  }
}

// CP: token columns of a consumer thread, a quarter of the tokens (a compile-time number, so that a slice is one straight
// piece of code: with a branch per 8 columns it took three times as long)
template <int KIND, int CP>
__global__ void __launch_bounds__(THREADS, 1) gemm5_kernel(const Args g) {
  asm volatile("griddepcontrol.launch_dependents;");
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr bool DS = KIND == G5_Q4K;
  constexpr int nt = 4 * CP, ub = unit_bytes(DS, nt);
  // slices per tensor-memory hand-off: two buffers of them (and Q4_K's two of minimum terms) in 512 columns
  constexpr int G = 16 * nt + (DS ? 2 * nt : 0) <= TMEM_COLS ? 8 : 8 * nt + (DS ? 2 * nt : 0) <= TMEM_COLS ? 4
                    : 4 * nt + (DS ? 2 * nt : 0) <= TMEM_COLS ? 2 : 1;
  static_assert(2 * G * nt + (DS ? 2 * nt : 0) <= TMEM_COLS, "tensor memory");
  const Smem S = smem_map(KIND, nt, g.b_stages);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const uint32_t bar0 = saddr(smem);
  const uint32_t a_full = bar0, a_empty = bar0 + 16, d_full = bar0 + 32, d_empty = bar0 + 48, b_full = bar0 + 64, b_empty = b_full + 8 * MAX_B;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
  auto wait = [&](uint32_t bar, uint32_t parity, uint32_t ns) -> bool { return wait_bar(bar, parity, abort_flag, ns); };

  // this CTA's units
  const int n_cta = gridDim.x;
  const int u0 = (int)((int64_t)blockIdx.x * g.n_units / n_cta), u1 = (int)((int64_t)(blockIdx.x + 1) * g.n_units / n_cta);

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(a_full + 8 * i, PROD_WARPS);
      mbar_init(a_empty + 8 * i, CONS_WARPS);   // (a drained superblock: its MMAs have completed too)
      mbar_init(d_full + 8 * i, 1);
      mbar_init(d_empty + 8 * i, CONS_WARPS);
    }
    for (int i = 0; i < MAX_B; ++i) {
      mbar_init(b_full + 8 * i, 1);
      mbar_init(b_empty + 8 * i, CONS_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) tmem_alloc(saddr(tmem_slot), TMEM_COLS);
  if (KIND == G5_IQ3S) {
    for (int i = tid; i < 512 * 8; i += THREADS) {
      const uint32_t v = g_grid[i >> 3];
      reinterpret_cast<uint4*>(smem + S.table)[i] = make_uint4(v, v, v, v);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp < PROD_WARPS) {
    // ------------------------------------------------------------------------------------ producers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(WORK_REGS));
    Ring ra = {0u, 0u};
    bool alive = true;
    if constexpr (KIND == G5_IQ3S) {
      const int gq = lane & 7, t = lane >> 3, rl = 4 * gq + t;
      auto record = [&](const Unit& at) -> const uint8_t* {
        const int row0 = at.rt * TR + 16 * warp;
        return row0 < g.nrows ? g.w + (int64_t)row0 * g.row_bytes + (int64_t)at.sb * 1760 : nullptr;
      };
      Rec3 cur = {}, nxt = {};
      Unit ahead(g, u0);
      const uint8_t* p = u0 < u1 ? record(ahead) : nullptr;
      if (p) cur.load(p, rl, gq);
      for (int u = u0; u < u1; ++u) {
        ahead.next(g);
        const uint8_t* pn = u + 1 < u1 ? record(ahead) : nullptr;
        if (pn) {
          nxt.load(pn, rl, gq);
          // the record two further on (of the same rows, or past them: a hint)
          if (lane < 14 && u + 3 < u1 && ahead.sb + 2 < g.nsb) asm volatile("prefetch.global.L2 [%0];" ::"l"(pn + 2 * 1760 + 128 * lane));
        }
        alive = wait(a_empty + 8 * ra.i, ra.ph ^ 1u, 100);
        if (!alive) break;
        uint8_t* a = smem + S.a + ra.i * a_stage(KIND);
        if (p) decode_iq3s(cur, a, reinterpret_cast<float*>(a + 8 * SL_A), smem + S.table, warp, gq, t, lane);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy stores -> tensor-core reads
        __syncwarp();
        if (lane == 0) mbar_arrive(a_full + 8 * ra.i);
        ra.next(A_STAGES);
        cur = nxt;
        p = pn;
      }
    } else {
      const int r = tid & 127, hf = tid >> 7;
      Unit ahead(g, u0);
      if (u0 < u1) fetch_raw<KIND>(g, ahead, smem + S.raw, tid);
      cp_async_commit();
      for (int u = u0; u < u1; ++u) {
        cp_async_wait<0>();
        asm volatile("bar.sync 1, %0;" ::"n"(PROD_THREADS) : "memory");   // everyone's pieces of u; everyone is done with u - 1
        ahead.next(g);
        if (u + 1 < u1) fetch_raw<KIND>(g, ahead, smem + S.raw + ((u + 1 - u0) & 1) * raw_bytes(KIND), tid);
        cp_async_commit();
        alive = alive && wait(a_empty + 8 * ra.i, ra.ph ^ 1u, 100);   // (after a wait has given up every thread still passes the barriers)
        if (alive) {
          const uint8_t* b = smem + S.raw + ((u - u0) & 1) * raw_bytes(KIND) + r * raw_row(KIND);
          uint8_t* a = smem + S.a + ra.i * a_stage(KIND);
          float* f = reinterpret_cast<float*>(a + 8 * SL_A);
          if (KIND == G5_IQ4XS) decode_iq4xs(b, a, f, r, hf);
          else decode_q4k(b, a, f, f + 8 * TR, a + 8 * SL_A + 9 * TR * 4, r, hf);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncwarp();
        if (alive && lane == 0) mbar_arrive(a_full + 8 * ra.i);
        ra.next(A_STAGES);
      }
      cp_async_wait<0>();
    }
  } else if (warp >= MMA_WARP) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(IDLE_REGS));
    if (warp == COPY_WARP) {
      // ---------------------------------------------------------------------------------- activation units
      if (lane == 0) {
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the quantiser has finished
        Ring rb = {0u, 0u};
        Unit at(g, u0);
        bool alive = true;
        int n = 0;
        for (int u = u0; u < u1; ++u, ++n) {
          alive = wait(b_empty + 8 * rb.i, rb.ph ^ 1u, 100);
          if (!alive) break;
          mbar_expect_tx(b_full + 8 * rb.i, ub);
          bulk_g2s(saddr(smem + S.b) + rb.i * ub, g.xb + ((int64_t)at.tb * g.nsb + at.sb) * ub, ub, b_full + 8 * rb.i);
          rb.next(g.b_stages);
          at.next(g);
        }
        if (!alive) {
          // let the copies in flight land (bounded) before the CTA's shared memory goes away
          for (int i = n < g.b_stages ? n : g.b_stages; i > 0; --i) {
            const int k = n - i;
            for (int spin = 0; spin < (1 << 16) && !try_bar(b_full + 8 * (k % g.b_stages), (uint32_t)(k / g.b_stages) & 1u); ++spin) {}
          }
        }
      }
      __syncwarp();
    } else if (warp == MMA_WARP) {
      // ---------------------------------------------------------------------------------- MMA issue
      const uint32_t id = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(TR >> 4) << 24);   // s8 x s8 -> s32
      const uint32_t idm = (1u << 4) | ((uint32_t)(nt >> 3) << 17) | ((uint32_t)(TR >> 4) << 24);                           // f16 x f16 -> f32
      const bool one = elect_one();
      Ring ra = {0u, 0u}, rb = {0u, 0u}, rd = {0u, 0u};
      bool alive = true;
      for (int u = u0; u < u1 && alive; ++u) {
        alive = __all_sync(0xFFFFFFFFu, wait(a_full + 8 * ra.i, ra.ph, 0) && wait(b_full + 8 * rb.i, rb.ph, 0));
        if (!alive) break;
        const uint32_t as = saddr(smem + S.a) + ra.i * a_stage(KIND), bs = saddr(smem + S.b) + rb.i * ub;
        for (int s0 = 0; s0 < 8; s0 += G) {
          alive = __all_sync(0xFFFFFFFFu, wait(d_empty + 8 * rd.i, rd.ph ^ 1u, 0));
          if (!alive) break;
          tc_fence_after();
          const uint32_t d = tmem_base + rd.i * G * nt;
          for (int s = 0; s < G; ++s) {
            const uint64_t ad = smem_desc(as + (s0 + s) * SL_A, 128, 256), bd = smem_desc(bs + (s0 + s) * nt * 32, 128, 256);
            if (one) mma_i8(d + s * nt, ad, bd, id);
          }
          if (DS && s0 + G == 8) {
            const uint64_t ad = smem_desc(as + 8 * SL_A + 9 * TR * 4, 128, 256), bd = smem_desc(bs + nt * 288, 128, 256);
            if (one) mma_f16(tmem_base + 2 * G * nt + ra.i * nt, ad, bd, idm, 0u);
          }
          if (one) mma_commit(d_full + 8 * rd.i);
          rd.next(2);
        }
        ra.next(A_STAGES);
        rb.next(g.b_stages);
      }
    }
  } else {
    // ------------------------------------------------------------------------------------ consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(WORK_REGS));
    const int q4 = warp & 3, cg = (warp - CONS_WARP0) >> 2;
    const int r_in = 32 * q4 + lane;
    const uint32_t t_warp = tmem_base + ((uint32_t)(32 * q4) << 16) + (uint32_t)(cg * CP);
    constexpr int NC = (CP + 7) / 8;              // chunks of 8 columns (the last one may be 4)
    Ring ra = {0u, 0u}, rb = {0u, 0u}, rd = {0u, 0u};
    Unit at(g, u0);
    bool alive = true;
    float2 acc[CP / 2];
#pragma unroll
    for (int i = 0; i < CP / 2; ++i) acc[i] = make_float2(0.0f, 0.0f);
    int first = u0;    // first unit of the tile being summed
    for (int u = u0; u < u1; ++u) {
      alive = wait(a_full + 8 * ra.i, ra.ph, 40) && wait(b_full + 8 * rb.i, rb.ph, 40);   // the row factors and the token scales
      if (!alive) break;
      const float* f = reinterpret_cast<const float*>(smem + S.a + ra.i * a_stage(KIND) + 8 * SL_A) + r_in;
      const float* bd = reinterpret_cast<const float*>(smem + S.b + rb.i * ub + nt * 256) + cg * CP;
      for (int s0 = 0; s0 < 8; s0 += G) {
        alive = wait(d_full + 8 * rd.i, rd.ph, 20);
        if (!alive) break;
        tc_fence_after();
        const uint32_t t = t_warp + rd.i * G * nt;
        // chunk by chunk, the next chunk's load (of this slice or the next) in flight while one is scaled
        uint32_t c0[8], c1[8];
        ld8(t, c0);
#pragma unroll 1
        for (int s = 0; s < G; ++s) {
          const float fs = f[(s0 + s) * TR];
          const float2 f2 = make_float2(fs, fs), nf2 = make_float2(-MAGIC_F * fs, -MAGIC_F * fs);
          const float* bds = bd + (s0 + s) * nt;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            uint32_t(&v)[8] = (c & 1) ? c1 : c0;
            uint32_t(&w)[8] = (c & 1) ? c0 : c1;
            ld_wait(v);
            if (c + 1 < NC) ld8(t + s * nt + 8 * (c + 1), w);
            else if (NC % 2 == 0 && s + 1 < G) ld8(t + (s + 1) * nt, c0);
            if (8 * c + 8 <= CP) scale<8>(v, f2, nf2, bds + 8 * c, acc + 4 * c);
            else scale<4>(v, f2, nf2, bds + 8 * c, acc + 4 * c);
            if (c + 1 == NC && NC % 2 == 1 && s + 1 < G) ld8(t + (s + 1) * nt, c0);
          }
        }
        if (DS && s0 + G == 8) {
          const float fm = f[8 * TR];
          const uint32_t tm = t_warp + 2 * G * nt + ra.i * nt;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            ld8(tm + 8 * c, c0);
            ld_wait(c0);
#pragma unroll
            for (int i = 0; i < (8 * c + 8 <= CP ? 4 : 2); ++i) {
              acc[4 * c + i].x = fmaf(__uint_as_float(c0[2 * i]), fm, acc[4 * c + i].x);
              acc[4 * c + i].y = fmaf(__uint_as_float(c0[2 * i + 1]), fm, acc[4 * c + i].y);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(d_empty + 8 * rd.i);
        rd.next(2);
      }
      if (!alive) break;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(a_empty + 8 * ra.i);
        mbar_arrive(b_empty + 8 * rb.i);
      }
      ra.next(A_STAGES);
      rb.next(g.b_stages);
      if (at.sb == g.nsb - 1 || u == u1 - 1) {
        const int row = at.rt * TR + r_in, tok0 = at.tb * nt + cg * CP;
        if (u - first == g.nsb - 1) {
          // the whole tile is this CTA's
          const int n = min(CP, g.m - tok0);
          const int64_t y0 = (int64_t)tok0 * g.ldy + row;
          if (row < g.nrows) {
            if (g.y_dtype == GSQ_BF16) store_cols<__nv_bfloat16, CP>((__nv_bfloat16*)g.y + y0, g.ldy, acc, n);
            else if (g.y_dtype == GSQ_F16) store_cols<__half, CP>((__half*)g.y + y0, g.ldy, acc, n);
            else store_cols<float, CP>((float*)g.y + y0, g.ldy, acc, n);
          }
        } else {
          const int64_t slot = 2 * (int64_t)blockIdx.x + (first == u0 ? 0 : 1);
          store_cols<float, CP>(g.part + (slot * nt + cg * CP) * TR + r_in, TR, acc, CP);
        }
        first = u + 1;
#pragma unroll
        for (int i = 0; i < CP / 2; ++i) acc[i] = make_float2(0.0f, 0.0f);
      }
      at.next(g);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, TMEM_COLS);
}

template <typename... KA, typename... A>
static int launch_pdl(void (*kern)(KA...), dim3 grid, int threads, int smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
  return GSQ_OK;
}

template <int KIND, int CP>
static int launch_t(const Args& g, int n_cta, cudaStream_t st) {
  static std::atomic<bool> configured[64];
  int dev = 0;
  GSQ_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return GSQ_ERR_UNSUPPORTED;
  if (!configured[dev]) {
    GSQ_CUDA_TRY(cudaFuncSetAttribute(gemm5_kernel<KIND, CP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured[dev] = true;
  }
  return launch_pdl(gemm5_kernel<KIND, CP>, dim3((unsigned)n_cta), THREADS, smem_map(KIND, g.nt, g.b_stages).total, st, g);
}
template <int KIND>
static int launch_kind(const Args& g, int n_cta, cudaStream_t st) {
  switch (g.nt / 4) {
    case 4: return launch_t<KIND, 4>(g, n_cta, st);
    case 8: return launch_t<KIND, 8>(g, n_cta, st);
    case 12: return launch_t<KIND, 12>(g, n_cta, st);
    case 16: return launch_t<KIND, 16>(g, n_cta, st);
    case 20: return launch_t<KIND, 20>(g, n_cta, st);
    case 24: return launch_t<KIND, 24>(g, n_cta, st);
    case 28: return launch_t<KIND, 28>(g, n_cta, st);
    case 32: return launch_t<KIND, 32>(g, n_cta, st);
    default: return GSQ_ERR_UNSUPPORTED;
  }
}
static int error_flag(int* flag) {
  GSQ_CUDA_TRY(cudaMemcpyFromSymbol(flag, g_error, sizeof(int)));
  return GSQ_OK;
}

}  // namespace g5
}  // namespace gsq
