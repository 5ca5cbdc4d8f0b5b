// The GEMM of the two-step product with exact integer slice sums (sm_100a: tcgen05 kind::f16, cta_group::2), for the types
// whose kernels of few rows have them: Q6_K, IQ3_S in GGUF order, Q2_K, IQ1_M. Operands as in gsq_gemm4.cu, but the
// activations are the bare quants: weights integer sub-scale x value (Q6_K: exact pair of planes), so that tensor memory
// holds S = sum over 32 values of sub * w * q, an integer below 2^24 (Q6_K: at most 128 * 32 * 127 * 32), whatever the order.
// The consumers scale in fp32, as those kernels do:
//     t += d_x[token, slice] * S      over the 8 slices of a superblock
//     acc += d[row, superblock] * t   over at most INT_PART superblocks (longer K: in parts, gsq_gemm4.cu's sum_parts)
// Two levels and short parts because every fp32 sum over n terms rounds n times: error against 64 bits, 2-norm, 1024 to
// 17408 columns 0.67e-7 to 0.95e-7, the kernels of few rows 0.69e-7 to 1.08e-7; scaled products accumulated in tensor memory,
// whose adder cuts off, 7e-7. For Q2_K and IQ1_M, whose kernel of few rows is the most exact (0.65e-7 at 1024 columns), t
// covers 4 slices and the sum over K carries its rounding error along: 0.55e-7 to 0.81e-7. Q2_K's minimums are 8 more sums per
// superblock, over the slice's two groups of m * (sum of q), scaled by -dmin the same way.
//
// A pair of CTAs owns 256 weight rows x nt tokens, 128 at most: two (three) fp32 numbers per result in the consumers'
// registers, and tensor memory for two pairs of slices (four up to 64 tokens).
//   warp 0        copies: k-blocks, `stages` deep; d_x, d and dmin of a superblock, 3 deep
//   warp 1        CTA 0: MMA issue, two slices (a k-block) at a time; CTA 1: reports each landed stage to CTA 0
//   warps 4..19   scaling: four warps per tensor-memory lane quarter, a quarter of the most tokens each
// What bounds it: no unit is full (Q6_K 5120 x 17408, 512 tokens: tensor pipe 44 %, issue 53 %, shared memory 36 %, L2 31 %). By
// clock64 stamps, taken when tensor memory was read by 16x256b loads, a k-block of 128 tokens took 1200 cycles, its operands (40 KB)
// were in after about 1050 and the tensor pipe needs 512; the loads of today took 7 us of 235 off this kernel. 8 consumer warps took
// 1450 cycles (one row a thread) and 1250 (four). The case: 331 us with expansion and sum, scaled products (two planes, 256
// tokens a block) 325, few-row launches 861.
// Every wait is bounded and raises the device flag instead of hanging.
#include <cuda_fp16.h>

#include "gsq_pair.cuh"
#include "gsq_planes.cuh"

namespace gsq {
namespace pl {

constexpr int S_THREADS = 640, S_CONS = 16;      // consumer warps
constexpr int S_IDLE_REGS = 64, S_CONS_REGS = 104;   // 128 x 64 + 512 x 104 = the 640 x 96 the block is launched with
constexpr int DX_SLOTS = 3;
constexpr int D_SLOTS = 4;          // most pairs of slices in tensor memory (2 above 64 tokens)
// tokens of a consumer warp: a quarter of the largest block
__host__ __device__ constexpr int warp_tokens(bool comp) { return (comp ? INT_NT_COMP : INT_NT) / 4; }

struct SliceArgs {
  const uint8_t *a, *ta, *b, *tb;
  const float *dw, *dm, *dx;
  void* y;
  int y_dtype;
  int64_t ldy;
  int nrows, m;
  int nsb, nt, n_tb, n_rp;
  int splits;
  float* part;
  int stages;
};

// Tensor memory -> registers in the layout of 16 rows x 4 columns per 2 registers: lane l holds column l % 4 of row l / 4 and of
// row l / 4 + 8. A thread then has a quarter of the tokens of four rows (two loads, 16 tensor-memory lanes each) instead of
// all tokens of one, and reads a quarter of the scales from shared memory: with one row a thread (32 x 32b) these reads, 128 of
// 16 bytes per slice, took as long as the tensor-memory loads, 560 cycles a slice together. Tensor memory gives an SM 512 bytes
// a cycle in this shape, 905 in that of 32 x 32b, but 256 in that of 8 columns per 4 registers (16 x 256b): 256 cycles for the
// 128 x 128 sums of a slice instead of 128, and with it Q6_K 5120 x 17408, 512 tokens, took 352 us, in this shape 344 (331 with the sum
// of the parts as it is now).
__device__ __forceinline__ void tmem_rows16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x128b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]),
        "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ void tmem_rows16(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x128b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr)
               : "memory");
}
template <int N>
__device__ __forceinline__ void pin(uint32_t (&v)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+r"(v[i]), "+r"(v[i + 1]), "+r"(v[i + 2]), "+r"(v[i + 3]), "+r"(v[i + 4]), "+r"(v[i + 5]), "+r"(v[i + 6]), "+r"(v[i + 7]));
}

// Results of a thread: tokens 4 i + lane % 4 of its four rows (8 apart), acc[2 * i + h] rows 2 h and 2 h + 1; y at its first
// token and row, `n` tokens from there, `rows` rows.
template <int ACC, typename T>
__device__ __forceinline__ void store_results(T* y, int64_t ldy, const float2 (&acc)[ACC], int n, int rows) {
#pragma unroll
  for (int i = 0; i < ACC / 2; ++i) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (4 * i < n) {
        if (16 * h < rows) store_out<T>(y + 16 * h, acc[2 * i + h].x);
        if (16 * h + 8 < rows) store_out<T>(y + 16 * h + 8, acc[2 * i + h].y);
      }
    }
    y += 4 * ldy;
  }
}

// acc += t * f with the rounding error of the sum carried along in e (Kahan). An infinite sum
// stays infinite: its error, which would be NaN, is cut to a number.
__device__ __forceinline__ void add_carried(float2& acc, float2& e, const float2& t, const float2& f) {
  const float2 minus = make_float2(-1.0f, -1.0f);
  const float2 y = __ffma2_rn(t, f, e), s = __fadd2_rn(acc, y);
  const float2 lost = __ffma2_rn(__ffma2_rn(acc, minus, s), minus, y);
  e = make_float2(fminf(fmaxf(lost.x, -1e35f), 1e35f), fminf(fmaxf(lost.y, -1e35f), 1e35f));
  acc = s;
}

// AP: planes of the weight operand; TP: 1 = a term unit per superblock (Q2_K's minimums); COMP: half a superblock at a time
// goes to a sum over all of K that carries its rounding error along
template <int AP, int TP, bool COMP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(S_THREADS, 1) gemm6_kernel(const SliceArgs g) {
  constexpr int FOLD = COMP ? 2 : 4;   // pairs of slices
  constexpr int WT = warp_tokens(COMP), ACC = WT / 2;   // tokens of a warp; pairs of results (rows 8 apart) of a thread
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t crank = cluster_ctarank();
  const int nth = g.nt >> 1;
  const uint32_t b_bytes = (uint32_t)nth * (KB * 2), a_bytes = AP * A_TILE, stage_bytes = a_bytes + b_bytes;
  const uint32_t tb_bytes = (uint32_t)nth * 32, t_bytes = TP ? 4096 + 8 * tb_bytes : 0;   // (fit into a stage)
  const uint32_t dx_bytes = (uint32_t)g.nt * 32, slot_bytes = dx_bytes + (1 + TP) * 512;   // d_x of a superblock, then d (and -dmin) of 128 rows
  const int n_stages = g.stages;
  const uint32_t d_cols = g.nt <= INT_NT / 2 ? INT_NT / 2 : INT_NT, d_slots = G_TMEM / (2 * d_cols);   // columns of a slice, pairs of slices
  constexpr int PER_SB = 4 + TP;    // stages of a superblock

  const uint32_t bar0 = saddr(smem);
  const uint32_t full = bar0, empty = full + 8 * MAX_STAGES, peer = empty + 8 * MAX_STAGES, d_full = peer + 8 * MAX_STAGES,
                 d_empty = d_full + 8 * D_SLOTS, dx_full = d_empty + 8 * D_SLOTS, dx_empty = dx_full + 8 * DX_SLOTS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + 512);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 516);
  const uint32_t st0 = saddr(smem + SMEM_HEAD), dx0 = st0 + n_stages * stage_bytes;
  const uint8_t* const dx_smem = smem + SMEM_HEAD + n_stages * stage_bytes;

  if (tid == 0) {
    *abort_flag = 0;
    for (int i = 0; i < MAX_STAGES; ++i) {
      mbar_init(full + 8 * i, 1);     // this CTA's copies of the stage have landed
      mbar_init(empty + 8 * i, 1);    // the MMAs that read the stage have completed
      mbar_init(peer + 8 * i, 1);     // (CTA 0) CTA 1's stage has landed
    }
    for (int i = 0; i < D_SLOTS; ++i) {
      mbar_init(d_full + 8 * i, 1);
      mbar_init(d_empty + 8 * i, 2 * S_CONS);
    }
    for (int i = 0; i < DX_SLOTS; ++i) {
      mbar_init(dx_full + 8 * i, 1);
      mbar_init(dx_empty + 8 * i, S_CONS);
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
  // one part of K after the other, so that the token blocks of a row tile run side by side and share its weights in L2
  const int tiles = g.n_rp * g.n_tb;
  auto place = [&](int item, int& rp, int& tb, int& sb0, int& sb1) {
    const int split = item / tiles;
    int all0, all1;
    place_item(item - split * tiles, 1, g.nsb, g.n_tb, g.n_rp, rp, tb, all0, all1);
    sb0 = split * g.nsb / g.splits;
    sb1 = (split + 1) * g.nsb / g.splits;
  };
  // the operands are written by the kernels before this one
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp < CONS_WARP0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S_IDLE_REGS));
    if (warp == 0 && lane == 0) {
      // ------------------------------------------------------------------------------------ copies
      Cursor c = {0u, 0u}, x = {0u, 0u};
      uint32_t n_loaded = 0, n_dx = 0;
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        const int64_t rt = 2 * rp + crank;
        const uint8_t* as = g.a + (rt * nkb + 4 * sb0) * (int64_t)a_bytes;
        const uint8_t* bs = g.b + (((int64_t)tb * nkb + 4 * sb0) * 2 + crank) * b_bytes;
        for (int sb = sb0; sb < sb1 && alive; ++sb) {
          alive = wait_bar(dx_empty + 8 * x.i, x.ph ^ 1u, abort_flag);
          if (!alive) break;
          const uint32_t to = dx0 + x.i * slot_bytes, xbar = dx_full + 8 * x.i;
          mbar_expect_tx(xbar, slot_bytes);
          bulk_g2s(to, g.dx + ((int64_t)tb * g.nsb + sb) * (8 * g.nt), dx_bytes, xbar);
          bulk_g2s(to + dx_bytes, g.dw + (rt * g.nsb + sb) * TR, 512, xbar);
          if (TP) bulk_g2s(to + dx_bytes + 512, g.dm + (rt * g.nsb + sb) * TR, 512, xbar);
          x.next(DX_SLOTS);
          ++n_dx;
          for (int kb = 0; kb < PER_SB; ++kb) {
            alive = wait_bar(empty + 8 * c.i, c.ph ^ 1u, abort_flag);
            if (!alive) break;
            const uint32_t dst = st0 + c.i * stage_bytes, bar = full + 8 * c.i;
            if (kb < 4) {
              mbar_expect_tx(bar, stage_bytes);
              bulk_g2s(dst, as, a_bytes, bar);
              bulk_g2s(dst + a_bytes, bs, b_bytes, bar);
              as += a_bytes;
              bs += 2 * b_bytes;
            } else {
              mbar_expect_tx(bar, t_bytes);
              bulk_g2s(dst, g.ta + (rt * g.nsb + sb) * 4096, 4096, bar);
              bulk_g2s(dst + 4096, g.tb + (((int64_t)tb * g.nsb + sb) * 2 + crank) * (8 * tb_bytes), 8 * tb_bytes, bar);
            }
            c.next(n_stages);
            ++n_loaded;
          }
        }
      }
      if (!alive) {
        // a wait gave up: let the copies in flight land (bounded) before the CTA's shared memory goes away
        auto drain = [](uint32_t bars, uint32_t loaded, uint32_t slots) {
          for (uint32_t i = loaded < slots ? loaded : slots; i > 0; --i) {
            const uint32_t k = loaded - i;
            for (int spin = 0; spin < (1 << 16) && !try_bar(bars + 8 * (k % slots), (k / slots) & 1u); ++spin) {}
          }
        };
        drain(full, n_loaded, n_stages);
        drain(dx_full, n_dx, DX_SLOTS);
      }
    } else if (warp == 1 && lane == 0 && crank != 0) {
      // ------------------------------------------------------------------------------------ CTA 1: stages to report
      Cursor c = {0u, 0u};
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        for (int i = 0; i < PER_SB * (sb1 - sb0) && alive; ++i) {
          alive = wait_bar(full + 8 * c.i, c.ph, abort_flag);
          if (!alive) break;
          arrive_remote(mapa(peer + 8 * c.i, 0u));
          c.next(n_stages);
        }
      }
    } else if (warp == 1 && crank == 0) {
      // ------------------------------------------------------------------------------------ CTA 0: MMA issue
      const uint32_t id = (1u << 4) | ((uint32_t)(g.nt >> 3) << 17) | ((uint32_t)(2 * TR >> 4) << 24);   // f16 x f16 -> f32, K-major
      const bool one = elect_one();
      Cursor c = {0u, 0u}, rd = {0u, 0u};
      bool alive = true;
      for (int item = pair; item < n_items && alive; item += n_pairs) {
        int rp, tb, sb0, sb1;
        place(item, rp, tb, sb0, sb1);
        for (int i = 0; i < PER_SB * (sb1 - sb0) && alive; ++i) {
          const int kb = i % PER_SB;
          alive = __all_sync(0xFFFFFFFFu, wait_bar(full + 8 * c.i, c.ph, abort_flag) && wait_bar(peer + 8 * c.i, c.ph, abort_flag));
          if (!alive) break;
          tc_fence_after();
          const uint32_t as = st0 + c.i * stage_bytes;
          // (descriptors before the branch of one lane: inside it every instruction would first move its operands there, 90
          // cycles each)
          const uint64_t ad = desc_sw128(as), bd = desc_sw128(as + a_bytes);
          if (!TP || kb < 4) {
            alive = __all_sync(0xFFFFFFFFu, wait_bar(d_empty + 8 * rd.i, rd.ph ^ 1u, abort_flag));
            if (!alive) break;
            tc_fence_after();
            const uint32_t d0 = tmem_base + rd.i * (2 * d_cols), d1 = d0 + d_cols;
            if (one) {
#pragma unroll
              for (int k = 0; k < 2 * AP; ++k)
                mma_f16_pair(d0, ad + (k >> 1) * (A_TILE >> 4) + 2 * (k & 1), bd + 2 * (k & 1), id, k > 0);
#pragma unroll
              for (int k = 0; k < 2 * AP; ++k)
                mma_f16_pair(d1, ad + (k >> 1) * (A_TILE >> 4) + 4 + 2 * (k & 1), bd + 4 + 2 * (k & 1), id, k > 0);
              commit_both(empty + 8 * c.i);
              commit_both(d_full + 8 * rd.i);
            }
            rd.next(d_slots);
          } else {
            const uint64_t td = smem_desc(as, 128, 256);
            uint64_t ud = smem_desc(as + 4096, 128, 256);
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {
              alive = __all_sync(0xFFFFFFFFu, wait_bar(d_empty + 8 * rd.i, rd.ph ^ 1u, abort_flag));
              if (!alive) break;
              tc_fence_after();
              const uint32_t d0 = tmem_base + rd.i * (2 * d_cols), d1 = d0 + d_cols;
              const uint64_t u1 = ud + (tb_bytes >> 4);
              if (one) {
                mma_f16_pair(d0, td, ud, id, 0u);
                mma_f16_pair(d1, td, u1, id, 0u);
                if (j == 3) commit_both(empty + 8 * c.i);
                commit_both(d_full + 8 * rd.i);
              }
              ud = u1 + (tb_bytes >> 4);
              rd.next(d_slots);
            }
          }
          c.next(n_stages);
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------------------------ consumers
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S_CONS_REGS));
    const int q4 = warp & 3, tok_w = ((warp - CONS_WARP0) >> 2) * WT;   // lane quarter, first token
    const int r_in = 32 * q4 + (lane >> 2), t_in = tok_w + (lane & 3);   // first row of the tile, first token of the thread
    const uint32_t t_warp = tmem_base + ((uint32_t)(32 * q4) << 16) + (uint32_t)tok_w;
    const uint32_t d_empty0 = mapa(d_empty, 0u);
    Cursor rd = {0u, 0u}, x = {0u, 0u};
    bool alive = true;
    for (int item = pair; item < n_items && alive; item += n_pairs) {
      int rp, tb, sb0, sb1;
      place(item, rp, tb, sb0, sb1);
      float2 acc[ACC], err[COMP ? ACC : 1];
#pragma unroll
      for (int i = 0; i < ACC; ++i) acc[i] = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int i = 0; i < (COMP ? ACC : 1); ++i) err[i] = make_float2(0.0f, 0.0f);
      for (int sb = sb0; sb < sb1 && alive; ++sb) {
        alive = wait_bar(dx_full + 8 * x.i, x.ph, abort_flag);
        if (!alive) break;
        const uint8_t* slot = dx_smem + x.i * slot_bytes;
#pragma unroll 1
        for (int part = 0; part < (1 + TP) * (4 / FOLD) && alive; ++part) {
          float2 t[ACC];
#pragma unroll
          for (int i = 0; i < ACC; ++i) t[i] = make_float2(0.0f, 0.0f);
#pragma unroll 1
          for (int j = 0; j < FOLD; ++j) {
            alive = wait_bar(d_full + 8 * rd.i, rd.ph, abort_flag);
            if (!alive) break;
            tc_fence_after();
            // the pair of slices has left tensor memory: its place may be overwritten
            auto release = [&] {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) arrive_remote(d_empty0 + 8 * rd.i);
            };
            if (tok_w >= g.nt) {
              release();
            } else {
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                const uint32_t ta = t_warp + rd.i * (2 * d_cols) + s * d_cols;
                // (tokens 4 i + lane % 4 lie side by side: gsq_planes.cu)
                const uint8_t* ds = slot + (((2 * (part * FOLD + j) + s) & 7) * g.nt + tok_w + 4 * (lane & 3)) * 4;
                float4 d[WT / 16];
#pragma unroll
                for (int i = 0; i < WT / 16; ++i) d[i] = *reinterpret_cast<const float4*>(ds + 64 * i);
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                  uint32_t v[WT / 2];
                  tmem_rows16(ta + ((uint32_t)(16 * hh) << 16), v);
                  tmem_ld_wait();
                  pin(v);
                  if (s == 1 && hh == 1) release();
                  // t += S * d_x: two registers per 4 columns, rows 16 hh + l / 4 and + 8
#pragma unroll
                  for (int i = 0; i < WT / 4; ++i) {
                    const float4& q = d[i >> 2];
                    const float dx = (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w;
                    t[2 * i + hh] = __ffma2_rn(make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), make_float2(dx, dx), t[2 * i + hh]);
                  }
                }
              }
            }
            rd.next(d_slots);
          }
          const float* f = reinterpret_cast<const float*>(slot + dx_bytes + (TP && part >= 4 / FOLD ? 512 : 0)) + r_in;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 scale = make_float2(f[16 * h], f[16 * h + 8]);
#pragma unroll
            for (int i = 0; i < ACC / 2; ++i) {
              if (COMP) add_carried(acc[2 * i + h], err[COMP ? 2 * i + h : 0], t[2 * i + h], scale);
              else acc[2 * i + h] = __ffma2_rn(t[2 * i + h], scale, acc[2 * i + h]);
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(dx_empty + 8 * x.i);
        x.next(DX_SLOTS);
      }
      if (alive) {
        const int row = (2 * rp + (int)crank) * TR + r_in, tok = tb * g.nt + t_in;
        const int n = min(g.nt - t_in, g.m - tok), rows = g.nrows - row;
        const int64_t to = (int64_t)tok * g.ldy + row;
        if (g.splits > 1) store_results(g.part + ((int64_t)(item / tiles) * g.m + tok) * g.nrows + row, g.nrows, acc, n, rows);
        else if (g.y_dtype == GSQ_BF16) store_results((__nv_bfloat16*)g.y + to, g.ldy, acc, n, rows);
        else if (g.y_dtype == GSQ_F16) store_results((__half*)g.y + to, g.ldy, acc, n, rows);
        else store_results((float*)g.y + to, g.ldy, acc, n, rows);
      }
    }
  }
  tc_fence_before();
  cluster_sync_all();   // no arrival of the peer is still on its way to this CTA's barriers, no MMA reads its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, G_TMEM);
}

// ---------------------------------------------------------------------------------------------

template <int AP, int TP, bool COMP>
static int launch_gemm6(SliceArgs& g, int sm_count, cudaStream_t st) {
  static std::atomic<int> max_pairs[64];
  const int stage = AP * A_TILE + g.nt / 2 * (KB * 2), dx = DX_SLOTS * (g.nt * 32 + (1 + TP) * 512);
  static_assert(!TP || 4096 + 8 * 32 * INT_NT / 2 <= AP * A_TILE + INT_NT / 2 * KB * 2, "a term unit fits into a stage");
  g.stages = (SMEM_MAX - SMEM_HEAD - dx) / stage;
  if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
  return launch_pairs(gemm6_kernel<AP, TP, COMP>, S_THREADS, g, max_pairs, (int64_t)g.n_rp * g.n_tb * g.splits, SMEM_HEAD + g.stages * stage + dx, sm_count, st);
}

int gemm6_launch(const Plan& p, uint8_t* scratch, int64_t rows, int64_t m, void* y, int y_dtype, int64_t ldy, int sm_count, cudaStream_t st) {
  SliceArgs g;
  g.a = scratch + p.a;
  g.ta = scratch + p.ta;
  g.b = scratch + p.b;
  g.tb = scratch + p.tb;
  g.dw = reinterpret_cast<const float*>(scratch + p.dw);
  g.dm = reinterpret_cast<const float*>(scratch + p.dm);
  g.dx = reinterpret_cast<const float*>(scratch + p.dx);
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
  g.part = reinterpret_cast<float*>(scratch + p.part);
  if (p.kind == K_Q2K) return launch_gemm6<1, 1, true>(g, sm_count, st);
  if (p.kind == K_IQ1M) return launch_gemm6<1, 0, true>(g, sm_count, st);
  return a_planes(p.kind) == 2 ? launch_gemm6<2, 0, false>(g, sm_count, st) : launch_gemm6<1, 0, false>(g, sm_count, st);
}

}  // namespace pl

int gemm6_error_flag(int* flag) {
  GSQ_CUDA_TRY(cudaMemcpyFromSymbol(flag, pl::pair_error, sizeof(int)));
  return GSQ_OK;
}

}  // namespace gsq
