// Operand layout of the two-step tensor-core product (gsq_expand.cu, gsq_planes.cu -> gsq_gemm4.cu, gsq_gemm6.cu) and the geometry all
// three agree on. Everything is fp16, K-major, in tiles of 64 values of K ("k-blocks", 4 per superblock), stored in
// global memory exactly as the tensor cores read them from shared memory, so that a stage is filled by plain bulk copies:
// 8-row groups of 1024 bytes, row r of a group at r * 128, its 16-byte chunk c (8 values) at ((c ^ r) * 16) -- the
// 128-byte swizzle of the matrix descriptor.
#pragma once
#include "gsq_common.cuh"

namespace gsq {
namespace pl {

enum Kind {
  K_Q4K = 0, K_IQ4XS = 1, K_IQ3S_PACKED = 2, K_Q6K_PACKED = 3, K_IQ3S = 4, K_Q6K = 5,
  K_Q2K = 6, K_IQ2XXS = 7, K_IQ2XS = 8, K_IQ2S = 9, K_IQ3XXS = 10, K_IQ1M = 11, K_NONE = 12
};

constexpr int TR = 128;         // weight rows of a tile (one CTA of a pair)
constexpr int KB = 64;          // values of K per k-block
constexpr int A_TILE = TR * KB * 2;
constexpr int MAX_NT = 256;     // most tokens of a block
constexpr int INT_NT = 128;     // the same of the form with integer slice sums (gsq_gemm6.cu)
constexpr int INT_NT_COMP = 64; // ... where the sum over K carries its rounding error along
constexpr int INT_PART = 12;    // most superblocks that it adds up in one sum, where that does not carry its error along

// fp16 planes of the weight operand: 2 for Q6_K, whose sub-scale times value reaches 4096 and needs 13 bits
__host__ __device__ constexpr int a_planes(int kind) { return kind == K_Q6K || kind == K_Q6K_PACKED ? 2 : 1; }
// planes of per-superblock extra columns (16 of them): Q4_K's minimum and correction terms, Q2_K's minimums
__host__ __device__ constexpr int t_planes(int kind) { return kind == K_Q4K || kind == K_Q2K ? 1 : 0; }
// Types whose kernels of few rows keep exact integer sums up to the fp32 scaling: so does their two-step product
// (gsq_gemm6.cu). Error against 64 bits, 2-norm over 1024 to 17408 columns: scaled products in two planes 4e-7 to 7e-7, the
// kernels of few rows 0.7e-7 to 1.1e-7. (The other low-bit types' few-row kernels truncate integer divisions as the
// reference's do, 1e-5 to 5e-5: two planes, 6e-7, are the more exact.)
__host__ __device__ constexpr bool int_sums(int kind) {
  return kind == K_Q6K || kind == K_Q6K_PACKED || kind == K_IQ3S || kind == K_Q2K || kind == K_IQ1M;
}

// (repacked weights: whole 16-row records, which the expanding kernel reads and writes as such; Q4_K and IQ4_XS have one
// layout, whatever the flag says, as in the kernels of fewer rows)
inline int kind_of(int ggml_type, int packed, int64_t rows) {
  if (ggml_type == GSQ_TYPE_Q4_K) return K_Q4K;
  if (ggml_type == GSQ_TYPE_IQ4_XS) return K_IQ4XS;
  if (packed && rows % 16 != 0) return K_NONE;
  switch (ggml_type) {
    case GSQ_TYPE_IQ3_S: return packed ? K_IQ3S_PACKED : K_IQ3S;
    case GSQ_TYPE_Q6_K: return packed ? K_Q6K_PACKED : K_Q6K;
    case GSQ_TYPE_Q2_K: return packed ? K_NONE : K_Q2K;
    case GSQ_TYPE_IQ2_XXS: return packed ? K_NONE : K_IQ2XXS;
    case GSQ_TYPE_IQ2_XS: return packed ? K_NONE : K_IQ2XS;
    case GSQ_TYPE_IQ2_S: return packed ? K_NONE : K_IQ2S;
    case GSQ_TYPE_IQ3_XXS: return packed ? K_NONE : K_IQ3XXS;
    case GSQ_TYPE_IQ1_M: return packed ? K_NONE : K_IQ1M;
    default: return K_NONE;
  }
}// ... with a sum over K that carries its rounding error along: the types whose kernel of few rows is the most exact
__host__ __device__ constexpr bool int_comp(int kind) { return kind == K_Q2K || kind == K_IQ1M; }

// How X is quantised: as the 128-value blocks with fp32 d or with half (d, sum x), or as block_q8_1 (half d). The same
// per type as in the kernels that serve it at fewer rows.
enum Form { F_D4 = 0, F_DS4 = 1, F_Q81 = 2 };
__host__ __device__ constexpr int form_of(int kind) {
  return kind == K_Q4K ? F_DS4 : kind == K_IQ4XS || kind == K_IQ3S_PACKED ? F_D4 : F_Q81;
}

// Sizes and places (bytes from the scratch buffer's start) of one product's operands.
struct Plan {
  int kind, hu;              // hu: planes of scaled products (1 = rounded, 2 = hi + lo); 0: the bare quants (int_sums)
  int nt, n_tb;              // tokens per block (a multiple of 16), blocks
  int splits;                // parts that K is cut into (few tiles: partial sums in fp32, then their sum)
  int nsb, nkb;
  int64_t chunk_rows;        // weight rows expanded and multiplied at a time (a multiple of 256)
  size_t a, dw, dm, ta, b, tb, inv, dx, part, total;
};
int make_plan(Plan* p, int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int hu);   // gsq_gemm4.cu

}  // namespace pl
}  // namespace gsq
