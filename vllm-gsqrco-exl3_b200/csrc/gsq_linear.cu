// gsq_linear: the whole product for callers that hand over X as it is (fp32 / fp16 / bf16) -- what the reference's
// ops that quantise for themselves do inside one call (lcpp_mul_mat_q, lcpp_mul_mat_mma_k, lcpp_mul_mat_iq3_packed:
// plugin/vllm_gguf_plugin/csrc/lcpp_shim.cu:626-671, 753-909). The activation quantiser and its output layout are
// chosen together with the kernel: 128-value blocks [K/128][M] for the small-batch tensor-core kernel and the
// lockstep GEMM, operand-ordered tiles for the prefill GEMM, 36-byte blocks for the dp4a kernel.
#include "gsq_common.cuh"

namespace gsq {

// gsq_mmv.cu
bool mmv_applies(int ggml_type, int packed, int64_t rows, int64_t m);
int mmv_rows_columns(int64_t m);
size_t mmv_rows_bytes(int ggml_type, int64_t m, int64_t k);
bool mmv_rows_wins(int ggml_type, int64_t rows, int64_t m, int64_t k);
int quantize_rows_host(const void* x, int x_dtype, int64_t m, int mc, int64_t k, int64_t stride, int ggml_type, void* out, void* stream);
bool mmv_raw_applies(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int vec);
int mmv_host(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* xq, int x_layout,
             int64_t m, int64_t k, void* y, int y_dtype, int64_t y_row_stride, void* stream, int* dump,
             const gsq_peer_reduce* pr = nullptr, int x_dtype = GSQ_BF16,
             int64_t x_row_stride = 0);
// gsq_gemm2.cu
bool gemm2_applies(int ggml_type, int packed, int64_t rows);
size_t gemm2_tile_bytes(int64_t m, int64_t k, int ggml_type);
int gemm2_host(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x_tiles, int64_t m,
               int64_t k, void* y, int y_dtype, int64_t y_row_stride, void* stream);
// gsq_gemm3.cu
bool gemm3_applies(int ggml_type, int packed, int64_t rows);
size_t gemm3_tile_bytes(int64_t m, int64_t k);
int gemm3_host(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x_tiles, int64_t m,
               int64_t k, void* y, int y_dtype, int64_t y_row_stride, void* stream);
// gsq_gemm5.cu
bool gemm5_applies(int ggml_type, int packed, int64_t rows, int64_t m);
size_t gemm5_scratch_bytes(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k);
int gemm5_linear(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype, int64_t m, int64_t k,
                 int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* scratch, void* stream);
// gsq_gemm4.cu
bool gemm4_applies(int ggml_type, int packed, int64_t rows);
size_t gemm4_scratch_bytes(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int hu);
int gemm4_linear(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype, int64_t m, int64_t k,
                 int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* scratch, int hu, void* stream);
// gsq_gemv.cu
int gemv_raw_host(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype, int64_t m, int64_t k,
                  int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* stream);
// gsq_quantize.cu
int quantize_tiles_host(const void* x, int x_dtype, int64_t m, int64_t k, int64_t stride, int layout, void* out, void* stream);
// gsq_gemm.cu
int* gemm_dump_pointer();
int gemm_variant();

static size_t align256(size_t v) { return (v + 255) / 256 * 256; }

static int g_prefill_precision = GSQ_PREFILL_ROUNDED;

// Repacked weights are records of 16 rows: no kernel takes a part of one.
static bool ragged(int ggml_type, int packed, int64_t rows) {
  return packed && (ggml_type == GSQ_TYPE_IQ3_S || ggml_type == GSQ_TYPE_Q6_K) && rows % 16 != 0;
}

// The kernels of a product above the small-batch tensor-core kernel's rows (or of a type or shape it does not serve).
enum Way {
  W_PLANES1,    // two steps, operands expanded to fp16: one plane of scaled activations (rounded)
  W_PLANES2,    // the same at fp32 accuracy: the activations as hi + lo, or bare quants and integer slice sums (gsq_gemm6.cu)
  W_IQ3_INT,    // gsq_gemm3.cu: fp16 operands, integer slice sums
  W_I8,         // gsq_gemm2.cu: int8 prefill GEMM
  W_BATCH,      // gsq_gemm5.cu: up to 256 rows, int8 operands decoded in the kernel, work cut evenly over the SMs
  W_LOCKSTEP,   // gsq_gemm.cu: 64-token tiles, split K
  W_MMV_LOOP,   // repacked Q6_K: the small-batch kernel, 48 rows per launch
  W_GEMV_LOOP   // GGUF-order blocks: the dp4a kernels, 8 rows per launch
};

// The fewest activation rows from which the two-step product takes the place of repeated launches of the small-batch
// kernels. Where the two cross, us two steps / launches (weights cycled through HBM; profiles/two_step_thresholds.txt):
//   Q6_K repacked (48 rows a launch)  97: 512 x 1024 15.2 / 19.8 (at 96 rows 14.9 / 14.3), 8192 x 8192 113.2 / 113.8 (112.2 / 94.8),
//                                     5120 x 17408 150 / 166 (151 / 143); 113 rows for tall weights of some size: 17408 x 5120
//                                     148 / 142 (97 rows 146 / 131), 12288 x 8192 167 / 165 (112 rows), but 9216 x 5120 97 rows 78 / 97;
//                                     81 where the third 16-row group of a launch costs more than the expansion: 5120 x 5120 (88
//                                     rows) 44.2 / 49.5, 4096 x 4096 30.9 / 35.0, but 2048 x 2048 20.7 / 18.9, 17408 x 2560 71 / 62;
//                                     49 where a launch has few rows of long K: 2048 x 8192 29.7 / 31.1 (64 rows 30.5 / 32.7, 96 rows
//                                     32.2 / 42.3), 1024 x 17408 39.7 / 40.8 (64 rows 39.9 / 46.0), 1024 x 5120 21.1 / 21.7.
//                                     The steps are coarse; cells of the sweep more than 4 % off: two steps too late for 512 x 8192
//                                     (64 to 96 rows 21.3 / 23.3 to 22.4 / 26.3), 9216 x 2560 and 9216 x 5120 (88, 96 rows 38 / 41,
//                                     77 / 82) and 17408 x 12800 (97 to 112 rows 364 / 412 to 365 / 428), too early for 34816 x 5120
//                                     (128 to 144 rows 316 / 274 to 363 / 309) and 151936 x 5120 (144 rows 1529 / 1452)
//   Q6_K, IQ3_S in GGUF order (8)     25: 512 x 1024 16 / 21 and 15 / 32, 17408 x 5120 148 / 281 and 95 / 176
//   Q2_K                              25: 5120 x 5120 47 / 70, 17408 x 5120 120 / 155; 512 x 1024 22 / 18, at 40 rows 23 / 26
//   IQ1_M                             12: 5120 x 5120 32 / 40, 17408 x 5120 81 / 89; 1024 x 2048 16.5 / 13.9, at 17 rows 17.4 / 18.9
//   the others                        9: 2048 x 8192 22 / 36 (IQ2_XXS) to 23 / 34 (IQ2_S); tall weights 78 / 75 (IQ2_S
//                                     17408 x 5120), at 12 rows 78 / 87; IQ2_S 2048 x 2048 14.8 / 13.6, at 12 rows 14.8 / 15.7
static int two_step_rows(int ggml_type, bool q6_packed, int64_t rows, int64_t k) {
  const int64_t values = rows * k;
  switch (ggml_type) {
    case GSQ_TYPE_Q6_K:
      if (!q6_packed) return 25;
      if (rows > 8192) return values > (48 << 20) ? 113 : 97;
      if (values > (4 << 20) && rows <= 2048 && k >= 5120) return 49;
      return values > (4 << 20) && values <= (32 << 20) ? 81 : 97;
    case GSQ_TYPE_IQ3_S: return 25;
    case GSQ_TYPE_Q2_K: return values <= (1 << 20) ? 33 : 25;
    case GSQ_TYPE_IQ1_M: return values <= (4 << 20) ? 17 : 12;
    default: return rows > 8192 || (ggml_type == GSQ_TYPE_IQ2_S && values <= (4 << 20)) ? 12 : 9;
  }
}

// small: the scratch has no room for expanded weights: the forms that need none instead, none less exact
static Way choose_way(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, bool small) {
  const int variant = gemm_variant();
  const bool dump = gemm_dump_pointer() != nullptr;   // (per-slice integer sums: only the integer forms have them)
  if (variant == 10 && !dump && gemm5_applies(ggml_type, packed, rows, m)) return W_BATCH;
  if (gemm2_applies(ggml_type, packed, rows)) {
    // Repacked IQ3_S, IQ4_XS, Q4_K. The prefill forms from 256 tokens on, and from 128 where the weight alone gives half
    // an SM count of row tiles; the int8 one, where integer sums are asked for, from 512 and 192. Below, the kernel with
    // integer sums and evenly cut work (100 rows, us, it / the lockstep kernel: IQ3_S 17408 x 5120 82 / 158, IQ4_XS
    // 5120 x 17408 90 / 261, Q4_K 2048 x 2048 17 / 21).
    const bool tall = (rows + 127) / 128 >= 74, iq3 = gemm3_applies(ggml_type, packed, rows);
    const bool big3 = m >= 256 || (m >= 128 && tall), big = m >= 512 || (m >= 192 && tall);
    if (variant == 3 || variant >= 5 || (variant == 0 && big3)) {
      int planes = g_prefill_precision == GSQ_PREFILL_ROUNDED ? 1 : g_prefill_precision == GSQ_PREFILL_SPLIT && iq3 ? 2 : 0;
      if (variant == 5 || variant == 9) planes = ggml_type == GSQ_TYPE_Q4_K ? 1 : 2;
      if (variant == 6 || variant == 8) planes = 1;
      if (variant == 7 || dump) planes = 0;
      if (planes && !(planes == 1 && small)) return planes == 1 ? W_PLANES1 : W_PLANES2;
      if (iq3) return W_IQ3_INT;
    }
    if (variant == 3 || variant == 4 || variant >= 5 || (variant == 0 && big)) return W_I8;
    return variant == 0 && !dump && gemm5_applies(ggml_type, packed, rows, m) ? W_BATCH : W_LOCKSTEP;
  }
  const bool q6_packed = ggml_type == GSQ_TYPE_Q6_K && packed && rows % 16 == 0;
  // Q6_K, IQ3_S in GGUF order and the low-bit types: the two steps once they cost less than the repeated launches of the
  // small-batch kernels (48 or 8 rows each), no less exact than those, unless they are asked for.
  if (!small && !dump && g_prefill_precision != GSQ_PREFILL_INTEGER && gemm4_applies(ggml_type, packed, rows) &&
      m >= two_step_rows(ggml_type, q6_packed, rows, k))
    return W_PLANES2;
  return q6_packed ? W_MMV_LOOP : W_GEMV_LOOP;
}

// Whether the small-batch tensor-core kernel is tried first. It serves 1..48 rows; for the types in GGUF order, whose
// decoding it repeats per lane, the kernel with evenly cut work takes over from 33 rows on where it is the faster one (us,
// small-batch kernel / evenly cut work, 33 and 48 rows):
//   * IQ4_XS: on weights so tall or large that the first one has no even plan: 60000 x 5120 154 / 153, 34816 x 12800 217 / 215,
//     5120 x 32768 94 / 91, but 34816 x 5120 78 / 94, 17408 x 5120 43 / 53, 5120 x 17408 52.9 / 54.8, 512 x 1024 7.9 / 8.9. To
//     16 M values the activations' size decides, as callers of gsq_route know it; that is not where the two cross (2048 x 8192,
//     40 to 48 rows: 18.2 / 22.8 to 18.3 / 22.9, and the second one runs).
//   * Q4_K: from 40 M values on, 17408 x 5120 52.7 / 50.4 and 54.3 / 50.8, 5120 x 12800 47 / 42, with long K from 20 M on,
//     2048 x 17408 32.4 / 31.6; but 7168 x 5120 26.0 / 28.0 and 26.6 / 28.3, 5120 x 8192 30.6 / 31.4, 1024 x 17408 26.0 / 28.2,
//     1024 x 2048 8.6 / 11.3. The line by size alone is early for some: 13312 x 4096 32.4 / 35.9, 9216 x 5120 33 rows 30.5 / 33.0
//     (48 rows 36.0 / 33.2), 4096 x 11264 32.6 / 34.1, 12288 x 5120 36.9 / 38.4.
static bool small_batch(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k) {
  if (gemm_variant() == 10 || !mmv_applies(ggml_type, packed, rows, m)) return false;
  if (m <= 32 || gemm_variant() != 0 || gemm_dump_pointer()) return true;
  if (ggml_type == GSQ_TYPE_IQ4_XS) return rows <= 40000 && (m * k <= 320000 || (rows * k > (16 << 20) && rows * k <= (100 << 20)));
  if (ggml_type == GSQ_TYPE_Q4_K) return rows * k <= (k <= 12288 ? 40 << 20 : 20 << 20);
  return true;
}

// GSQ_KERNEL_* of a gsq_linear call with the scratch it wants most
int linear_kernel(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k) {
  if (ragged(ggml_type, packed, rows)) return GSQ_KERNEL_NONE;
  if (small_batch(ggml_type, packed, rows, m, k)) return GSQ_KERNEL_MMV;
  switch (choose_way(ggml_type, packed, rows, m, k, false)) {
    case W_PLANES1:
    case W_PLANES2:
    case W_IQ3_INT:
    case W_I8: return GSQ_KERNEL_GEMM_PREFILL;
    case W_BATCH:
    case W_LOCKSTEP: return GSQ_KERNEL_GEMM;
    case W_MMV_LOOP: return GSQ_KERNEL_MMV;
    default: return GSQ_KERNEL_GEMV;
  }
}

static size_t way_scratch(Way way, int64_t rows, int64_t m, int64_t k, int ggml_type, int packed) {
  switch (way) {
    case W_PLANES1: return gemm4_scratch_bytes(ggml_type, packed, rows, m, k, 1);
    case W_PLANES2: return gemm4_scratch_bytes(ggml_type, packed, rows, m, k, 2);
    case W_IQ3_INT: return gemm3_tile_bytes(m, k);
    case W_I8: return gemm2_tile_bytes(m, k, ggml_type);
    case W_BATCH: return gemm5_scratch_bytes(ggml_type, packed, rows, m, k);
    case W_LOCKSTEP: return (size_t)(k / 128) * (size_t)m * 144;
    default: return (size_t)(k / 32) * (size_t)m * 36;
  }
}

}  // namespace gsq

extern "C" int gsq_prefill_precision(int mode) {
  const int old = gsq::g_prefill_precision;
  if (mode >= GSQ_PREFILL_ROUNDED && mode <= GSQ_PREFILL_INTEGER) gsq::g_prefill_precision = mode;
  return old;
}

static size_t linear_bytes(int64_t rows, int64_t m, int64_t k, int ggml_type, int packed, bool small) {
  using namespace gsq;
  if (m <= 0 || k <= 0 || rows <= 0 || ragged(ggml_type, packed, rows)) return 0;
  const Way way = choose_way(ggml_type, packed, rows, m, k, small);
  size_t b = way_scratch(way, rows, m, k, ggml_type, packed);
  if (small && gemm2_applies(ggml_type, packed, rows) && choose_way(ggml_type, packed, rows, m, k, false) == W_PLANES1) {
    // one fp16 plane of activations (and Q4_K's block sums): room for any of the forms of the default precision
    const size_t plane = gemm3_tile_bytes(m, k) + (ggml_type == GSQ_TYPE_Q4_K ? (size_t)((m + 255) / 256) * (k / 256) * 8192 : 0);
    b = b > plane ? b : plane;
  }
  // (the small-batch kernel takes 128-value blocks, and may decline the shape)
  size_t mmq = small_batch(ggml_type, packed, rows, m, k) ? (size_t)(k / 128) * (size_t)m * 144 : 0;
  if (mmq && !small && mmv_rows_wins(ggml_type, rows, m, k) && mmv_rows_bytes(ggml_type, m, k) > mmq) mmq = mmv_rows_bytes(ggml_type, m, k);
  b = b > mmq ? b : mmq;
  return align256(b > 0 ? b : 1);
}
extern "C" size_t gsq_linear_scratch_bytes(int64_t rows, int64_t m, int64_t k, int ggml_type, int packed) {
  const size_t small = linear_bytes(rows, m, k, ggml_type, packed, true), full = linear_bytes(rows, m, k, ggml_type, packed, false);
  return small < full ? small : full;
}
extern "C" size_t gsq_linear_workspace_bytes(int64_t rows, int64_t m, int64_t k, int ggml_type, int packed) {
  return linear_bytes(rows, m, k, ggml_type, packed, false);
}

extern "C" int gsq_linear(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x,
                          int x_dtype, int64_t m, int64_t k, int64_t x_row_stride, void* y, int y_dtype,
                          int64_t y_row_stride, void* scratch, size_t scratch_bytes, void* stream) {
  using namespace gsq;
  if (m == 0 || rows == 0) return GSQ_OK;
  if (m < 0 || rows < 0 || k <= 0 || k % 256 != 0 || !w || !x || !y) return GSQ_ERR_UNSUPPORTED;
  const int bs = block_bytes(ggml_type);
  if (bs == 0 || row_bytes != (k / 256) * bs || ragged(ggml_type, packed, rows)) return GSQ_ERR_UNSUPPORTED;
  if (y_dtype != GSQ_F32 && y_dtype != GSQ_F16 && y_dtype != GSQ_BF16) return GSQ_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < gsq_linear_scratch_bytes(rows, m, k, ggml_type, packed)) return GSQ_ERR_SCRATCH;
  const int layout = gsq_q8_layout_for_type(ggml_type);
  int rc;
  // 1..48 rows: the small-batch tensor-core kernel on 128-value blocks, where it serves the type and the shape fits
  if (small_batch(ggml_type, packed, rows, m, k)) {
    if (!gemm_dump_pointer() && mmv_raw_applies(ggml_type, packed, rows, m, k, 0)) {
      rc = mmv_host(w, row_bytes, rows, ggml_type, packed, x, 3, m, k, y, y_dtype, y_row_stride, stream, nullptr, nullptr, x_dtype, x_row_stride);
      if (rc != 1000) return rc;
    }
    const int mc = mmv_rows_columns(m);
    const bool in_rows = mmv_rows_wins(ggml_type, rows, m, k) && !gemm_dump_pointer() && scratch_bytes >= mmv_rows_bytes(ggml_type, m, k) &&
                         (uintptr_t)scratch % 16 == 0;
    rc = in_rows ? quantize_rows_host(x, x_dtype, m, mc, k, x_row_stride, ggml_type, scratch, stream)
                 : gsq_quantize_q8_1_mmq(x, x_dtype, m, k, x_row_stride, layout, scratch, stream);
    if (rc != GSQ_OK) return rc;
    rc = mmv_host(w, row_bytes, rows, ggml_type, packed, scratch, in_rows ? 4 : 1, m, k, y, y_dtype, y_row_stride, stream, gemm_dump_pointer());
    if (rc != 1000) return rc;  // 1000: declined, the activations of this shape do not fit its staging area
  }
  const Way way = choose_way(ggml_type, packed, rows, m, k, scratch_bytes < gsq_linear_workspace_bytes(rows, m, k, ggml_type, packed));
  const int64_t ysz = y_dtype == GSQ_F32 ? 4 : 2;
  switch (way) {
    case W_PLANES1:
    case W_PLANES2:
      return gemm4_linear(w, row_bytes, rows, ggml_type, packed, x, x_dtype, m, k, x_row_stride, y, y_dtype, y_row_stride, scratch,
                          way == W_PLANES1 ? 1 : 2, stream);
    case W_IQ3_INT:
      rc = quantize_tiles_host(x, x_dtype, m, k, x_row_stride, Q8_TILES_H16, scratch, stream);
      if (rc != GSQ_OK) return rc;
      return gemm3_host(w, row_bytes, rows, ggml_type, packed, scratch, m, k, y, y_dtype, y_row_stride, stream);
    case W_I8:
      rc = quantize_tiles_host(x, x_dtype, m, k, x_row_stride, layout, scratch, stream);
      if (rc != GSQ_OK) return rc;
      return gemm2_host(w, row_bytes, rows, ggml_type, packed, scratch, m, k, y, y_dtype, y_row_stride, stream);
    case W_BATCH:
      return gemm5_linear(w, row_bytes, rows, ggml_type, packed, x, x_dtype, m, k, x_row_stride, y, y_dtype, y_row_stride, scratch, stream);
    case W_LOCKSTEP:
      rc = gsq_quantize_q8_1_mmq(x, x_dtype, m, k, x_row_stride, layout, scratch, stream);
      if (rc != GSQ_OK) return rc;
      return gsq_mul_mat_q8(w, row_bytes, rows, ggml_type, packed, scratch, m, k, y, y_dtype, y_row_stride, nullptr, 0, stream);
    default: break;
  }
  // as many rows per launch as the kernel takes, on 36-byte blocks of the whole X
  rc = gsq_quantize_q8_1(x, x_dtype, m, k, x_row_stride, scratch, stream);
  if (rc != GSQ_OK) return rc;
  const int64_t step = way == W_MMV_LOOP ? 48 : gsq_mul_mat_vec_max_rows(ggml_type, packed);
  for (int64_t i = 0; i < m; i += step) {
    const int64_t c = m - i < step ? m - i : step;
    const uint8_t* xq = (const uint8_t*)scratch + i * (k / 32) * 36;
    uint8_t* yi = (uint8_t*)y + i * y_row_stride * ysz;
    if (way == W_MMV_LOOP) {
      rc = mmv_host(w, row_bytes, rows, ggml_type, packed, xq, 0, c, k, yi, y_dtype, y_row_stride, stream, nullptr);
      if (rc == 1000) return GSQ_ERR_TOO_LARGE;
    } else {
      rc = gsq_mul_mat_vec_q8(w, row_bytes, rows, ggml_type, packed, xq, c, k, yi, y_dtype, y_row_stride, stream);
    }
    if (rc != GSQ_OK) return rc;
  }
  return GSQ_OK;
}

extern "C" int gsq_linear_allreduce(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x,
                                    int x_dtype, int64_t m, int64_t k, int64_t x_row_stride, void* y, int y_dtype,
                                    int64_t y_row_stride, void* scratch, size_t scratch_bytes, const gsq_peer_reduce* pr,
                                    void* stream) {
  using namespace gsq;
  if (!pr || m <= 0 || m > 48 || rows <= 0 || k <= 0 || k % 256 != 0 || !w || !x || !y) return GSQ_ERR_UNSUPPORTED;
  const int bs = block_bytes(ggml_type);
  if (bs == 0 || row_bytes != (k / 256) * bs) return GSQ_ERR_UNSUPPORTED;
  if (y_dtype != GSQ_F32 && y_dtype != GSQ_F16 && y_dtype != GSQ_BF16) return GSQ_ERR_UNSUPPORTED;
  if (!scratch || scratch_bytes < gsq_linear_scratch_bytes(rows, m, k, ggml_type, packed)) return GSQ_ERR_SCRATCH;
  if (!mmv_applies(ggml_type, packed, rows, m)) return GSQ_ERR_UNSUPPORTED;
  int rc = gsq_quantize_q8_1_mmq(x, x_dtype, m, k, x_row_stride, gsq_q8_layout_for_type(ggml_type), scratch, stream);
  if (rc != GSQ_OK) return rc;
  rc = mmv_host(w, row_bytes, rows, ggml_type, packed, scratch, 1, m, k, y, y_dtype, y_row_stride, stream, nullptr, pr);
  return rc == 1000 ? GSQ_ERR_UNSUPPORTED : rc;   // 1000: the shape does not fit the kernel's staging area
}

extern "C" int gsq_linear_vec(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* x, int x_dtype,
                              int64_t m, int64_t k, int64_t x_row_stride, void* y, int y_dtype, int64_t y_row_stride, void* stream) {
  using namespace gsq;
  if (m == 0 || rows == 0) return GSQ_OK;
  if (m < 0 || m > 8 || rows < 0 || k <= 0 || k % 256 != 0 || !w || !x || !y) return GSQ_ERR_UNSUPPORTED;
  if (!mmv_raw_applies(ggml_type, packed, rows, m, k, 1)) {
    if (small_batch(ggml_type, packed, rows, m, k)) return GSQ_ERR_UNSUPPORTED;   // (that kernel on blocks)
    const int rc = gemv_raw_host(w, row_bytes, rows, ggml_type, packed, x, x_dtype, m, k, x_row_stride, y, y_dtype, y_row_stride, stream);
    return rc == GSQ_ERR_TOO_LARGE ? GSQ_ERR_UNSUPPORTED : rc;   // (X does not fit)
  }
  const int rc = mmv_host(w, row_bytes, rows, ggml_type, packed, x, 2, m, k, y, y_dtype, y_row_stride, stream, nullptr, nullptr, x_dtype,
                          x_row_stride);
  return rc == 1000 ? GSQ_ERR_UNSUPPORTED : rc;
}
