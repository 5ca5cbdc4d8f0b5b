// The GEMM of the two-step product (sm_100a: tcgen05 kind::f16, cta_group::2): y = x w^T from the fp16 operand tiles that
// gsq_expand.cu (weights: integer sub-scale times integer value) and gsq_planes.cu (activations: d * q * 2^e, one plane
// or hi + lo) have written. Tensor memory accumulates over one superblock (256 values of K); the consumers add
// C * factor[row, superblock] in fp32 registers, and multiply by 2^-e[token] at the end of K: the arithmetic of the
// quantised formats, with the only rounding of the operands that of hi (one-plane form).
//
// A pair of CTAs (cluster of 2) owns 256 weight rows x nt tokens (nt <= 256). Each CTA copies its own 128 rows of the
// weight operand and half of the tokens (bulk copies: the operand is stored as the tensor cores read it); the MMAs
// (M = 256) are issued by CTA 0. Per 64 values of K an SM takes in 16 KB of weights and at most 16 KB of activations per
// plane for 512 cycles of tensor work; nothing else uses its shared memory.
//   warp 0        copies, `stages` deep
//   warp 1        CTA 0: MMA issue; CTA 1: reports each landed stage to CTA 0
//   warps 4..11   read a superblock's sums (two warps per tensor-memory lane quarter, half of the tokens each) while the
//                 next superblock's are formed in the other half of tensor memory: 128 FMAs per thread and superblock of
//                 2048 cycles
// Pairs are persistent; items run in groups of 8 row tiles, token blocks inside, so that the pairs running at one time
// share both operands in L2. Every wait is bounded and raises the device flag instead of hanging.
#include <cuda_fp16.h>

#include "gsq_pair.cuh"
#include "gsq_planes.cuh"

namespace gsq {
namespace pl {

constexpr int MODEL_PAIRS = 74;                  // pairs of SMs the plan is made for

// k-blocks per stage: 128 values of K of the one-plane form, so that the MMA warp's waits and commits (about 400 cycles)
// stay behind the 1024 cycles of tensor work they belong to; 64 values of the other, which has two MMAs for each
__host__ __device__ constexpr int stage_kblocks(int hu) { return hu == 1 ? 2 : 1; }

struct GemmArgs {
  const uint8_t *a, *ta, *b, *tb;
  const float *dw, *inv;
  void* y;
  int y_dtype;
  int64_t ldy;
  int nrows, m;             // rows of this call, tokens
  int nsb, nt, n_tb, n_rp;  // superblocks, tokens per block, token blocks, pairs of row tiles
  int splits;               // > 1: item = a part of K of a tile, its fp32 sums go to part[split][token][rows]
  float* part;
  int stages;
};

// A row's n tokens (32 lanes: 32 neighbouring rows); lane l holds the reciprocal scales of tokens 4 l .. 4 l + 3.
template <typename T>
__device__ __forceinline__ void store_tokens(T* y, int64_t ldy, const float2 (&acc)[64], const float4& inv, int n, bool row_ok) {
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    if (4 * i >= n) break;
    const float s0 = __shfl_sync(0xFFFFFFFFu, inv.x, i), s1 = __shfl_sync(0xFFFFFFFFu, inv.y, i);
    const float s2 = __shfl_sync(0xFFFFFFFFu, inv.z, i), s3 = __shfl_sync(0xFFFFFFFFu, inv.w, i);
    if (row_ok) {
      store_out<T>(y, acc[2 * i].x * s0);
      if (4 * i + 1 < n) store_out<T>(y + ldy, acc[2 * i].y * s1);
      if (4 * i + 2 < n) store_out<T>(y + 2 * ldy, acc[2 * i + 1].x * s2);
      if (4 * i + 3 < n) store_out<T>(y + 3 * ldy, acc[2 * i + 1].y * s3);
    }
    y += 4 * ldy;
  }
}

template <int HU, int TP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G_THREADS, 1) gemm4_kernel(const GemmArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t crank = cluster_ctarank();
  const int nth = g.nt >> 1;
  constexpr int KS = stage_kblocks(HU);
  const uint32_t b_plane = (uint32_t)nth * (KB * 2), b_bytes = HU * b_plane, a_bytes = A_TILE;   // of one k-block
  const uint32_t ta_bytes = TP * 4096, tb_bytes = (uint32_t)(TP * nth * 32);
  const uint32_t b_off = KS * a_bytes, t_off = b_off + KS * b_bytes, stage_bytes = t_off + (TP ? TP * 8192 : 0);
  const int n_stages = g.stages;

  const uint32_t bar0 = saddr(smem);
  const uint32_t full = bar0, empty = full + 8 * MAX_STAGES, peer = empty + 8 * MAX_STAGES, d_full = peer + 8 * MAX_STAGES,
                 d_empty = d_full + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
  const uint32_t st0 = saddr(smem + SMEM_HEAD);

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < MAX_STAGES; ++i) {
      mbar_init(full + 8 * i, 1);     // this CTA's copies of the stage have landed
      mbar_init(empty + 8 * i, 1);    // the MMAs that read the stage have completed
      mbar_init(peer + 8 * i, 1);     // (CTA 0) CTA 1's stage has landed
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(d_full + 8 * i, 1);
      mbar_init(d_empty + 8 * i, 2 * CONS_WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(saddr(tmem_slot), G_TMEM);
  tc_fence_before();
  cluster_sync_all();   // the peer's barriers are initialised before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
  const int n_items = g.n_rp * g.n_tb * g.splits, nkb = 4 * g.nsb;
  auto place = [&](int item, int& rp, int& tb, int& sb0, int& sb1) { place_item(item, g.splits, g.nsb, g.n_tb, g.n_rp, rp, tb, sb0, sb1); };
  // the operands are written by the kernels before this one
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp < CONS_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(IDLE_REGS));
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------------------------ copies
      Cursor c = {0u, 0u};
      uint32_t n_loaded = 0;
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        const int64_t rt = 2 * rp + crank;
        const uint8_t* as = g.a + (rt * nkb + 4 * sb0) * (int64_t)a_bytes;
        const uint8_t* bs = g.b + (((int64_t)tb * nkb + 4 * sb0) * 2 + crank) * b_bytes;
        const uint8_t* tas = TP ? g.ta + (rt * g.nsb + sb0) * (int64_t)ta_bytes : nullptr;
        const uint8_t* tbs = TP ? g.tb + (((int64_t)tb * g.nsb + sb0) * 2 + crank) * tb_bytes : nullptr;
        for (int kb = 4 * sb0; kb < 4 * sb1; kb += KS) {
          alive = wait_bar(empty + 8 * c.i, c.ph ^ 1u, abort_flag);
          if (!alive) break;
          const uint32_t dst = st0 + c.i * stage_bytes, bar = full + 8 * c.i;
          const bool terms = TP && (kb & 3) == 0;
          mbar_expect_tx(bar, t_off + (terms ? ta_bytes + tb_bytes : 0u));
          bulk_g2s(dst, as, KS * a_bytes, bar);
#pragma unroll
          for (int i = 0; i < KS; ++i) bulk_g2s(dst + b_off + i * b_bytes, bs + i * 2 * b_bytes, b_bytes, bar);
          if (terms) {
            bulk_g2s(dst + t_off, tas, ta_bytes, bar);
            bulk_g2s(dst + t_off + ta_bytes, tbs, tb_bytes, bar);
            tas += ta_bytes;
            tbs += 2 * tb_bytes;
          }
          as += KS * a_bytes;
          bs += KS * 2 * b_bytes;
          c.next(n_stages);
          ++n_loaded;
        }
      }
      if (!alive) {
        // a wait gave up: let the copies in flight land (bounded) before the CTA's shared memory goes away
        const uint32_t n = n_loaded < (uint32_t)n_stages ? n_loaded : (uint32_t)n_stages;
        for (uint32_t i = n; i > 0; --i) {
          const uint32_t k = n_loaded - i, slot = k % n_stages, ph = (k / n_stages) & 1u;
          for (int spin = 0; spin < (1 << 16); ++spin) {
            uint32_t done;
            asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                         : "=r"(done) : "r"(full + 8 * slot), "r"(ph) : "memory");
            if (done) break;
          }
        }
      }
    } else if (warp == 1 && lane == 0 && crank != 0) {
      // ------------------------------------------------------------------------------------ CTA 1: stages to report
      Cursor c = {0u, 0u};
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        for (int kb = 4 * sb0; kb < 4 * sb1 && alive; kb += KS) {
          alive = wait_bar(full + 8 * c.i, c.ph, abort_flag);
          if (!alive) break;
          arrive_remote(mapa(peer + 8 * c.i, 0u));
          c.next(n_stages);
        }
      }
    } else if (warp == 1 && crank == 0) {
      // ------------------------------------------------------------------------------------ CTA 0: MMA issue
      // The whole warp walks the loop, so that descriptors and addresses stay in uniform registers (issued from a
      // one-lane branch every instruction first moved its operands there: ~90 cycles each); one lane issues.
      const uint32_t id = (1u << 4) | ((uint32_t)(g.nt >> 3) << 17) | ((uint32_t)(2 * TR >> 4) << 24);   // f16 x f16 -> f32, K-major
      const bool one = elect_one();
      Cursor c = {0u, 0u}, rd = {0u, 0u};
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        for (int sb = sb0; sb < sb1 && alive; ++sb) {
          alive = __all_sync(0xFFFFFFFFu, wait_bar(d_empty + 8 * rd.i, rd.ph ^ 1u, abort_flag));
          if (!alive) break;
          const uint32_t d = tmem_base + rd.i * 256;
#pragma unroll 1
          for (int kb = 0; kb < 4; kb += KS) {
            alive = __all_sync(0xFFFFFFFFu, wait_bar(full + 8 * c.i, c.ph, abort_flag) && wait_bar(peer + 8 * c.i, c.ph, abort_flag));
            if (!alive) break;
            tc_fence_after();
            const uint32_t as = st0 + c.i * stage_bytes, bs = as + b_off;
            const uint64_t ad = desc_sw128(as), bd = desc_sw128(bs);
            if (one) {
              uint32_t acc = kb > 0 ? 1u : 0u;
              if (TP && kb == 0) {
                const uint32_t ta = as + t_off, tb = ta + ta_bytes;
                mma_f16_pair(d, smem_desc(ta, 128, 256), smem_desc(tb, 128, 256), id, 0u);
                acc = 1u;
              }
              if (HU == 1) {
#pragma unroll
                for (int i = 0; i < KS; ++i) {
#pragma unroll
                  for (int k = 0; k < 4; ++k)
                    mma_f16_pair(d, ad + i * (A_TILE >> 4) + 2 * k, bd + i * (b_plane >> 4) + 2 * k, id, i || k ? 1u : acc);
                }
              } else {
                // per 32 values hi, then lo: the order in which a one-tile kernel with the same operands would add them
                const uint64_t bl = bd + (b_plane >> 4);
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                  mma_f16_pair(d, ad + 4 * s, bd + 4 * s, id, s ? 1u : acc);
                  mma_f16_pair(d, ad + 4 * s + 2, bd + 4 * s + 2, id, 1u);
                  mma_f16_pair(d, ad + 4 * s, bl + 4 * s, id, 1u);
                  mma_f16_pair(d, ad + 4 * s + 2, bl + 4 * s + 2, id, 1u);
                }
              }
              commit_both(empty + 8 * c.i);
              if (kb == 4 - KS) commit_both(d_full + 8 * rd.i);
            }
            c.next(n_stages);
          }
          rd.next(2);
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------------------------ consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONS_REGS));
    const int q4 = warp & 3, cg = (warp - CONS_WARP0) >> 2;
    const int r_in = 32 * q4 + lane;
    const uint32_t t_warp = tmem_base + ((uint32_t)(32 * q4) << 16) + (uint32_t)(cg * nth);
    const uint32_t d_empty0 = mapa(d_empty, 0u);
    Cursor rd = {0u, 0u};
    bool alive = true;
    for (int item = pair; item < n_items && alive; item += n_pairs) {
      int rp, tb, sb0, sb1;
      place(item, rp, tb, sb0, sb1);
      const int rt = 2 * rp + (int)crank, row = rt * TR + r_in;
      const float* dwp = g.dw + (int64_t)rt * g.nsb * TR + r_in;
      float2 acc[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) acc[i] = make_float2(0.0f, 0.0f);
      const int tok0 = tb * g.nt + cg * nth;
      const float4 inv = 4 * lane < nth ? __ldcg(reinterpret_cast<const float4*>(g.inv + tok0 + 4 * lane)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      float dw_next = __ldcg(dwp + sb0 * TR);
      for (int sb = sb0; sb < sb1; ++sb) {
        const float dw = dw_next;
        if (sb + 1 < sb1) dw_next = __ldcg(dwp + (sb + 1) * TR);
        alive = wait_bar(d_full + 8 * rd.i, rd.ph, abort_flag);
        if (!alive) break;
        tc_fence_after();
        const uint32_t t = t_warp + rd.i * 256;
        const float2 dw2 = make_float2(dw, dw);
        // 64 columns at a time: two loads of 32 in flight, one wait
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
          if (64 * ch < nth) {
            uint32_t v[64];
            tmem_ld32(t + 64 * ch, v);
            if (64 * ch + 32 < nth) tmem_ld32(t + 64 * ch + 32, v + 32);
            tmem_ld_wait();
            pin32(v);
            pin32(v + 32);
#pragma unroll
            for (int j = 0; j < 32; ++j)
              acc[32 * ch + j] = __ffma2_rn(make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), dw2, acc[32 * ch + j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) arrive_remote(d_empty0 + 8 * rd.i);
        rd.next(2);
      }
      if (alive) {
        const int n = min(nth, g.m - tok0);
        const int64_t at = (int64_t)tok0 * g.ldy + row;
        const bool row_ok = row < g.nrows;
        if (g.splits > 1) {
          const int64_t split = item % g.splits;
          store_tokens(g.part + (split * g.m + tok0) * g.nrows + row, g.nrows, acc, inv, n, row_ok);
        } else if (g.y_dtype == GSQ_BF16) store_tokens((__nv_bfloat16*)g.y + at, g.ldy, acc, inv, n, row_ok);
        else if (g.y_dtype == GSQ_F16) store_tokens((__half*)g.y + at, g.ldy, acc, inv, n, row_ok);
        else store_tokens((float*)g.y + at, g.ldy, acc, inv, n, row_ok);
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();   // no arrival of the peer is still on its way to this CTA's barriers, no MMA reads its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, G_TMEM);
}

// ---------------------------------------------------------------------------------------------

static int stage_bytes_of(const Plan& p) {
  return stage_kblocks(p.hu) * (A_TILE + p.hu * (p.nt / 2) * KB * 2) + t_planes(p.kind) * 8192;
}

template <int HU, int TP>
static int launch_gemm4(GemmArgs& g, int stage, int sm_count, cudaStream_t st) {
  static std::atomic<int> max_pairs[64];
  g.stages = (SMEM_MAX - SMEM_HEAD) / stage;
  if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
  return launch_pairs(gemm4_kernel<HU, TP>, G_THREADS, g, max_pairs, (int64_t)g.n_rp * g.n_tb * g.splits, SMEM_HEAD + g.stages * stage, sm_count, st);
}

static int gemm4_launch(const Plan& p, uint8_t* scratch, int64_t rows, int64_t m, void* y, int y_dtype, int64_t ldy, int sm_count,
                        cudaStream_t st) {
  GemmArgs g;
  g.a = scratch + p.a;
  g.ta = scratch + p.ta;
  g.b = scratch + p.b;
  g.tb = scratch + p.tb;
  g.dw = reinterpret_cast<const float*>(scratch + p.dw);
  g.inv = reinterpret_cast<const float*>(scratch + p.inv);
  g.y = y;
  g.y_dtype = y_dtype;
  g.ldy = ldy;
  g.nrows = (int)rows;
  g.m = (int)m;
  g.nsb = p.nsb;
  g.nt = p.nt;
  g.n_tb = p.n_tb;
  g.n_rp = (int)((rows + 255) / 256);
  g.splits = p.splits;
  g.part = (float*)(scratch + p.part);
  const int stage = stage_bytes_of(p);
  if (t_planes(p.kind)) return launch_gemm4<1, 1>(g, stage, sm_count, st);
  return p.hu == 2 ? launch_gemm4<2, 0>(g, stage, sm_count, st) : launch_gemm4<1, 0>(g, stage, sm_count, st);
}

// y = the sum of the parts, in their order; a thread takes V rows of a token (4 where rows and y allow it: 16-byte loads, all of
// a thread's in flight; with one row Q6_K 5120 rows x 512 tokens in 6 parts, 63 MB, took 19.6 us). Tokens are the grid's x: a
// prompt may have more than the 65535 blocks of y (row blocks of a call: 4096 at most, by the bound on expanded weights).
template <typename T, int V>
__global__ void __launch_bounds__(256) sum_parts_kernel(const float* __restrict__ part, T* __restrict__ y, int64_t m, int64_t rows, int64_t ldy,
                                                       int splits) {
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t row = ((int64_t)blockIdx.y * 256 + threadIdx.x) * V, tok = blockIdx.x;
  if (row >= rows) return;
  const float* p = part + tok * rows + row;
  if constexpr (V == 1) {
    float s = __ldcg(p);
    for (int i = 1; i < splits; ++i) s += __ldcg(p + i * m * rows);
    store_out<T>(y + tok * ldy + row, s);
  } else {
    float4 s = __ldcg(reinterpret_cast<const float4*>(p));
#pragma unroll 8
    for (int i = 1; i < splits; ++i) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p + i * m * rows));
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    alignas(16) T r[4];
    store_out<T>(r, s.x);
    store_out<T>(r + 1, s.y);
    store_out<T>(r + 2, s.z);
    store_out<T>(r + 3, s.w);
    if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4*>(y + tok * ldy + row) = *reinterpret_cast<const uint4*>(r);
    else *reinterpret_cast<uint2*>(y + tok * ldy + row) = *reinterpret_cast<const uint2*>(r);
  }
}

template <typename T>
static int launch_sum_parts(const Plan& p, const float* part, int64_t rows, int64_t m, T* y, int64_t ldy, cudaStream_t st) {
  const bool vec = rows % 4 == 0 && ldy % 4 == 0 && (uintptr_t)y % (4 * sizeof(T)) == 0;
  const int64_t per = vec ? 1024 : 256;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)m, (unsigned)((rows + per - 1) / per));
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  GSQ_CUDA_TRY(cudaLaunchKernelEx(&cfg, vec ? sum_parts_kernel<T, 4> : sum_parts_kernel<T, 1>, part, y, m, rows, ldy, p.splits));
  return GSQ_OK;
}
static int sum_parts(const Plan& p, const uint8_t* scratch, int64_t rows, int64_t m, void* y, int y_dtype, int64_t ldy, cudaStream_t st) {
  const float* part = reinterpret_cast<const float*>(scratch + p.part);
  if (y_dtype == GSQ_BF16) return launch_sum_parts(p, part, rows, m, (__nv_bfloat16*)y, ldy, st);
  if (y_dtype == GSQ_F16) return launch_sum_parts(p, part, rows, m, (__half*)y, ldy, st);
  return launch_sum_parts(p, part, rows, m, (float*)y, ldy, st);
}

// Tokens per block, blocks and parts of K of a product of n_rp pairs of row tiles and m tokens, by an estimate in SM
// cycles. A k-block costs the larger of its MMAs (2 cycles per token and plane product) and of bringing its operands into
// shared memory (about 40 bytes per cycle and SM when all pairs load); an item 4000 beyond that (pipeline fill, the last
// superblock's drain, stores); waves are whole. Splitting K writes and reads fp32 partial sums: 5000 for the extra kernel
// and their bytes at 2 KB per cycle.
static void choose_tiles(Plan* p, int64_t n_rp, int64_t rows, int64_t m) {
  const bool ints = int_sums(p->kind);
  const int ap = a_planes(p->kind), hu = ints ? 1 : p->hu, products = ints ? ap : hu, max_nt = !ints ? MAX_NT : int_comp(p->kind) ? INT_NT_COMP : INT_NT;
  const int parts = ints && !int_comp(p->kind) ? (p->nsb + INT_PART - 1) / INT_PART : 1;   // the least
  double best = 1e300;
  const int64_t first = (m + max_nt - 1) / max_nt;
  for (int64_t b = first; b <= first + 8 && (b == first || (m + b - 1) / b >= 48); ++b) {
    const int64_t t = ((m + b - 1) / b + 15) / 16 * 16, blocks = (m + t - 1) / t;
    double kblock = 2.0 * t * products, load = ap * 16384.0 + hu * 64.0 * t;
    if (ints) {
      // the chain of a k-block through the consumers (Q2_K: twice), and their scales
      const double cons = (1 + t_planes(p->kind)) * (2.5 * t + 900.0);
      kblock = cons > kblock ? cons : kblock;
      load += 8.0 * t + t_planes(p->kind) * (1024.0 + 32.0 * t);
    }
    kblock = (kblock > load / 40.0 ? kblock : load / 40.0) + 20.0;
    for (int s = parts; s <= (parts > 8 ? parts : 8) && (s == parts || p->nsb / s >= 4); ++s) {
      const double waves = (double)((n_rp * blocks * s + MODEL_PAIRS - 1) / MODEL_PAIRS);
      double cost = waves * (4.0 * ((p->nsb + s - 1) / s) * kblock + 4000.0);
      if (s > 1) cost += 5000.0 + (double)s * m * rows * 8.0 / 2048.0;
      if (cost < 0.97 * best) {
        best = cost;
        p->nt = (int)t;
        p->n_tb = (int)blocks;
        p->splits = s;
      }
    }
  }
}

int make_plan(Plan* p, int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int hu) {
  p->kind = kind_of(ggml_type, packed, rows);
  if (p->kind == K_NONE || rows <= 0 || m <= 0 || k <= 0 || k % 256 != 0) return GSQ_ERR_UNSUPPORTED;
  const bool ints = int_sums(p->kind);
  if (form_of(p->kind) == F_Q81) hu = ints ? 0 : 2;
  if (p->kind == K_Q4K) hu = 1;
  p->hu = hu;
  p->nsb = (int)(k / 256);
  p->nkb = 4 * p->nsb;
  const int ap = a_planes(p->kind), tp = t_planes(p->kind);
  const int64_t rows_pad = (rows + 255) / 256 * 256;
  // the expanded weights of a call (with the least of partial sums) are bounded (512 MB); taller ones go a chunk of rows at a time
  const int64_t per_row = (int64_t)ap * k * 2, parts = ints && !int_comp(p->kind) ? (p->nsb + INT_PART - 1) / INT_PART : 1;
  int64_t chunk = ((int64_t)512 << 20) / (per_row + (parts > 1 ? parts * m * 4 : 0)) / 256 * 256;
  if (chunk < 256) chunk = 256;
  p->chunk_rows = rows_pad < chunk ? rows_pad : chunk;
  choose_tiles(p, p->chunk_rows / 256, p->chunk_rows < rows ? p->chunk_rows : rows, m);
  auto up = [](size_t v) { return (v + 1023) / 1024 * 1024; };
  const size_t c = (size_t)p->chunk_rows, tokens = (size_t)p->nt * p->n_tb;
  size_t at = 0;
  p->a = at;
  at = up(at + c * (size_t)per_row);
  p->dw = at;
  at = up(at + c * p->nsb * 4);
  p->dm = at;
  if (ints && tp) at = up(at + c * p->nsb * 4);
  p->ta = at;
  at = up(at + (size_t)tp * c * p->nsb * 32);
  p->b = at;
  at = up(at + (size_t)(ints ? 1 : p->hu) * tokens * (size_t)k * 2);
  p->tb = at;
  at = up(at + (size_t)tp * tokens * p->nsb * 32 * (ints ? 8 : 1));
  p->inv = at;
  if (!ints) at = up(at + tokens * 4);
  p->dx = at;
  if (ints) at = up(at + tokens * (size_t)(k / 32) * 4);
  p->part = at;
  if (p->splits > 1) at = up(at + (size_t)p->splits * m * (size_t)(p->chunk_rows < rows ? p->chunk_rows : rows) * 4);
  p->total = at;
  return GSQ_OK;
}

int planes_host(const Plan& p, const void* x, int x_dtype, int64_t m, int64_t k, int64_t stride, uint8_t* scratch, cudaStream_t st);
int expand_host(const Plan& p, const uint8_t* w, int64_t row_bytes, int64_t rows, uint8_t* scratch, int sm_count, cudaStream_t st);
int gemm6_launch(const Plan& p, uint8_t* scratch, int64_t rows, int64_t m, void* y, int y_dtype, int64_t ldy, int sm_count, cudaStream_t st);

}  // namespace pl

int gemm6_error_flag(int* flag);   // gsq_gemm6.cu

int gemm4_error_flag(int* flag) {
  int a = 0, b = 0;
  GSQ_CUDA_TRY(cudaMemcpyFromSymbol(&a, pl::pair_error, sizeof(int)));
  const int rc = gemm6_error_flag(&b);
  *flag = a | b;
  return rc;
}

bool gemm4_applies(int ggml_type, int packed, int64_t rows) { return pl::kind_of(ggml_type, packed, rows) != pl::K_NONE; }

size_t gemm4_scratch_bytes(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int hu) {
  pl::Plan p;
  return pl::make_plan(&p, ggml_type, packed, rows, m, k, hu) == GSQ_OK ? p.total : 0;
}

// The whole product by the two steps; scratch: gemm4_scratch_bytes, 256-byte aligned.
int gemm4_linear(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype, int64_t m, int64_t k,
                 int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* scratch, int hu, void* stream) {
  if (rows > INT32_MAX || k > INT32_MAX || m > INT32_MAX - 512) return GSQ_ERR_TOO_LARGE;
  pl::Plan p;
  int rc = pl::make_plan(&p, ggml_type, packed, rows, m, k, hu);
  if (rc != GSQ_OK) return rc;
  DeviceInfo di;
  rc = device_info(&di);
  if (rc != GSQ_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ysz = y_dtype == GSQ_F32 ? 4 : 2;
  for (int64_t r0 = 0; r0 < rows && rc == GSQ_OK; r0 += p.chunk_rows) {
    const int64_t n = rows - r0 < p.chunk_rows ? rows - r0 : p.chunk_rows;
    rc = pl::expand_host(p, (const uint8_t*)w + r0 * row_bytes, row_bytes, n, (uint8_t*)scratch, di.sm_count, st);
    // (beside the first expansion: the order of these two launches matters, see planes_kernel)
    if (rc == GSQ_OK && r0 == 0) rc = pl::planes_host(p, x, x_dtype, m, k, x_row_stride, (uint8_t*)scratch, st);
    if (rc == GSQ_OK)
      rc = (pl::int_sums(p.kind) ? pl::gemm6_launch : pl::gemm4_launch)(p, (uint8_t*)scratch, n, m, (uint8_t*)y + r0 * ysz, y_dtype, y_row_stride,
                                                                        di.sm_count, st);
    if (rc == GSQ_OK && p.splits > 1) rc = pl::sum_parts(p, (const uint8_t*)scratch, n, m, (uint8_t*)y + r0 * ysz, y_dtype, y_row_stride, st);
  }
  return rc;
}

}  // namespace gsq
