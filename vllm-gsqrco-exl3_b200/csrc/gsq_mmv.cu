// Host side of the register-operand tensor-core product (gsq_mmv.cuh): which calls it serves, experiment settings, dispatch
// to the translation unit of the weight type.
#include "gsq_mmv.cuh"

namespace gsq {

static int g_mmv_mode = 0;      // 0 = use this kernel wherever it applies, 1 = never (the older kernels)
static int g_mmv_min_rows = 0;  // fewest activation rows served here; 0 = per type (see mmv_applies)
static int g_mmv_max_rows = 48; // most
int g_mmv_cluster = 0;   // experiments: 0 = choose, else 1, 2, 4 or 8
static unsigned long long* g_mmv_prof = nullptr;
int g_mmv_pdl = 2;       // programmatic stream serialisation: 0 off, 1 on, 2 + early start of the dependents where it pays, 3 + everywhere
int g_mmv_pf_first = 2;  // records requested from L2 ahead of the staging
int g_mmv_aligned = -1;  // experiments: -1 = choose, 0 / 1 = equal chunks / whole tiles per warp
int g_mmv_trace = 0;     // one line per launch plan on stderr

// shared with the dp4a kernel: whether a product lets the next kernels of a programmatic-launch chain start early
bool mmv_early_trigger() { return g_mmv_pdl >= 2; }

int mmv_launch_q4k(const MmvArgs& a, int x_layout, int sm_count, int max_smem, cudaStream_t st);   // gsq_mmv_q4k.cu
int mmv_errors_q4k(int* peer, int* copy);
int mmv_launch_iq4xs(const MmvArgs& a, int x_layout, int sm_count, int max_smem, cudaStream_t st);   // gsq_mmv_iq4xs.cu
int mmv_errors_iq4xs(int* peer, int* copy);
int mmv_launch_iq3s(const MmvArgs& a, int x_layout, int sm_count, int max_smem, cudaStream_t st);   // gsq_mmv_iq3s.cu
int mmv_errors_iq3s(int* peer, int* copy);
int mmv_launch_q6k(const MmvArgs& a, int x_layout, int sm_count, int max_smem, cudaStream_t st);   // gsq_mmv_q6k.cu
int mmv_errors_q6k(int* peer, int* copy);

// Whether (type, packed, m) may be served here (mmv_host can still decline a shape: MMV_DECLINED).
bool mmv_applies(int ggml_type, int packed, int64_t rows, int64_t m) {
  if ((g_mmv_mode == 1 && !(ggml_type == GSQ_TYPE_Q6_K && packed)) || m > 48 ||
      (m > g_mmv_max_rows && !(ggml_type == GSQ_TYPE_Q6_K && packed))) return false;
  // Below these row counts the dp4a GEMV is faster on the measured shapes (its start-up is shorter: no staging of
  // the activations, no cluster-wide sum); packed IQ3_S has no faster kernel at any count.
  int min_rows;
  switch (ggml_type) {
    case GSQ_TYPE_Q4_K: min_rows = 2; break;
    case GSQ_TYPE_IQ4_XS: min_rows = 4; break;
    case GSQ_TYPE_IQ3_S:
    case GSQ_TYPE_Q6_K:   // (repacked Q6_K has no other kernel: served here at every count)
      if (!packed || rows % 16 != 0) return false;
      min_rows = 1;
      break;
    default: return false;
  }
  if (ggml_type == GSQ_TYPE_Q6_K) return true;
  return m >= (g_mmv_min_rows > 0 ? g_mmv_min_rows : min_rows);
}

// Whether X itself (quantised while it is staged) may be served here: as block_q8_1 (vec) 1..8 rows, as block_q8_1_mmq
// 1..16. A quantiser kernel in front costs 1 to 2 us of GPU time and, where the host is what limits, 2.5 us of its time;
// quantising in every CTA costs about 0.5 us per 1000 values of a CTA's share. Level at 16000 values of X, with IQ3_S at 10000
// (GPU us, here / two kernels: Q6_K 5120 x 5120 1 row 10.6 / 11.3, 4 rows 11.0 / 11.4, 8 rows 12.0 / 11.8; Q4_K
// 17408 x 5120 2 rows 17.1 / 17.4, 4 rows 17.9 / 17.6; IQ3_S 17408 x 5120 1 row 18.2 / 18.7, 4 rows 18.9 / 18.6); on small
// products at 40000 (1024 x 5120 8 rows Q6_K 7.8 / 8.2), where the host's share counts too (1024 x 2048 called one by one
// 5.4 / 8.0).
bool mmv_raw_applies(int ggml_type, int packed, int64_t rows, int64_t m, int64_t k, int vec) {
  if (g_mmv_mode == 1 || m > (vec ? 8 : 16) || m > g_mmv_max_rows || m < g_mmv_min_rows) return false;
  const bool small = rows * k <= (8 << 20), iq3 = ggml_type == GSQ_TYPE_IQ3_S;
  if (m * k > (small ? 40960 : iq3 ? 10240 : 16384)) return false;
  switch (ggml_type) {
    case GSQ_TYPE_Q4_K:
    case GSQ_TYPE_IQ4_XS:
      // (at these row counts the dp4a kernel is faster, 8.0 / 11.9 us at 5120 x 5120, but for the launch that it costs)
      if (m < (ggml_type == GSQ_TYPE_Q4_K ? 2 : 4) && rows * k > (3 << 20)) return false;
      return !packed;
    case GSQ_TYPE_IQ3_S:
    case GSQ_TYPE_Q6_K: return packed && rows % 16 == 0;
    default: return false;
  }
}

// the arguments of a product, but for what its launch plan sets
static MmvArgs mmv_args(const void* w, int64_t row_bytes, int64_t rows, const void* xq, int64_t m, int64_t k, void* y, int y_dtype, int64_t y_row_stride,
                        int* dump, int x_dtype, int64_t x_row_stride) {
  MmvArgs a;
  a.w = (const uint8_t*)w;
  a.row_bytes = row_bytes;
  a.nrows = (int)rows;
  a.k = (int)k;
  a.xq = (const uint8_t*)xq;
  a.m = (int)m;
  a.y = y;
  a.y_dtype = y_dtype;
  a.ldy = y_row_stride;
  a.ntiles = (int)((rows + MMV_TR - 1) / MMV_TR);
  a.tiles_base = a.tiles_extra = a.tiles_round = 0;
  a.aligned = 0;
  a.xcap_kb = 0;
  a.dump = dump;
  a.prof = g_mmv_prof;
  a.pr_slots = nullptr;
  a.pr_flags = nullptr;
  a.pr_state = nullptr;
  a.pr_rank = 0;
  a.pr_world = 1;
  a.pr_slot_bytes = 0;
  a.x_dtype = x_dtype;
  a.x_stride = x_row_stride;
  a.x_vec = (uintptr_t)xq % 16 == 0 && (x_row_stride * (x_dtype == GSQ_F32 ? 4 : 2)) % 16 == 0;
  return a;
}

// x_layout: 0 = block_q8_1, 1 = block_q8_1_mmq. Returns MMV_DECLINED when the shape does not fit.
// x_layout 4: quantize_rows_host's. x_layout 2 / 3: xq is X itself (x_dtype, rows x_row_stride elements apart), up to 8 / 16 rows.
int mmv_host(const void* w, int64_t row_bytes, int64_t rows, int ggml_type, int packed, const void* xq, int x_layout,
             int64_t m, int64_t k, void* y, int y_dtype, int64_t y_row_stride, void* stream, int* dump,
             const gsq_peer_reduce* pr, int x_dtype, int64_t x_row_stride) {
  if (pr && (m == 0 || rows == 0)) return GSQ_ERR_UNSUPPORTED;   // every rank must launch: nothing to skip
  if (m == 0 || rows == 0) return GSQ_OK;
  if (m < 0 || m > 48 || rows < 0 || k <= 0 || k % 256 != 0 || !w || !xq || !y) return GSQ_ERR_UNSUPPORTED;
  if (rows > INT32_MAX || k > INT32_MAX) return GSQ_ERR_TOO_LARGE;
  const int bs = block_bytes(ggml_type);
  if (bs == 0 || row_bytes != (k / 256) * bs) return GSQ_ERR_UNSUPPORTED;
  if (y_dtype != GSQ_F32 && y_dtype != GSQ_F16 && y_dtype != GSQ_BF16) return GSQ_ERR_UNSUPPORTED;
  DeviceInfo di;
  const int rc = device_info(&di);
  if (rc != GSQ_OK) return rc;
  MmvArgs a = mmv_args(w, row_bytes, rows, xq, m, k, y, y_dtype, y_row_stride, dump, x_dtype, x_row_stride);
  if (x_layout == XL_ROWS && (dump || pr || (uintptr_t)xq % 16 != 0)) return GSQ_ERR_UNSUPPORTED;
  if ((x_layout == XL_XQ81 || x_layout == XL_XMMQ) && ((x_dtype != GSQ_F32 && x_dtype != GSQ_F16 && x_dtype != GSQ_BF16) || dump || pr)) return GSQ_ERR_UNSUPPORTED;
  if (pr) {
    const int64_t esz = y_dtype == GSQ_F32 ? 4 : 2;
    if (!pr->slots || !pr->flags || !pr->state || pr->world < 2 || pr->world > 8 || pr->rank < 0 || pr->rank >= pr->world ||
        pr->slot_bytes < ((m - 1) * y_row_stride + rows) * esz || pr->slot_bytes % 16 != 0 || dump)
      return GSQ_ERR_UNSUPPORTED;
    a.pr_slots = pr->slots;
    a.pr_flags = pr->flags;
    a.pr_state = pr->state;
    a.pr_rank = pr->rank;
    a.pr_world = pr->world;
    a.pr_slot_bytes = pr->slot_bytes;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if ((ggml_type == GSQ_TYPE_IQ3_S || ggml_type == GSQ_TYPE_Q6_K) && (!packed || rows % 16 != 0)) return MMV_DECLINED;
  switch (ggml_type) {
    case GSQ_TYPE_Q4_K: return mmv_launch_q4k(a, x_layout, di.sm_count, di.max_smem_optin, st);
    case GSQ_TYPE_IQ4_XS: return mmv_launch_iq4xs(a, x_layout, di.sm_count, di.max_smem_optin, st);
    case GSQ_TYPE_IQ3_S: return mmv_launch_iq3s(a, x_layout, di.sm_count, di.max_smem_optin, st);
    case GSQ_TYPE_Q6_K: return mmv_launch_q6k(a, x_layout, di.sm_count, di.max_smem_optin, st);
    default: return MMV_DECLINED;
  }
}

// weight values of which one launch for two products still serves the smaller of them
constexpr int64_t MMV_PAIR_VALUES = 96 << 20;

// Whether the pair serves two weights at m rows. One launch saves the smaller product its start, staging and last step and the
// wait for the larger one, 5 to 8 us, but gives both one cluster size and leaves the clusters of the product that ends first
// idle. Measured against two launches in a graph over 1892 cells of the four pairs of types, 19 pairs of row counts from 512 + 256 to
// 34816 + 34816, K 1024 to 17408, 1 to 8 rows (profiles/mmv_pair.txt): 28 % less on average. Where the smaller product alone takes
// 20 us and more the saving no longer covers the rest: 17408 + 17408 rows IQ3_S + IQ4_XS, 4 rows, K 17408 122.7 / 111.4 us, K 8192
// 61.4 / 59.8 (but K 5120, 89 M values, 41.6 / 43.3, and Q4_K + Q6_K 35.1 / 37.0). Below that line the pair loses on some
// weights of K 17408, at most 7 %, and nowhere to K 8192.
bool mmv_pair_serves(const gsq_weight* a, const gsq_weight* b, int64_t m) {
  if (m < 1 || m > 8 || !mmv_pair_types(a->ggml_type, b->ggml_type) || !mmv_applies(a->ggml_type, a->packed, a->rows, m) ||
      !mmv_applies(b->ggml_type, b->packed, b->rows, m))
    return false;
  const int64_t va = a->row_bytes / block_bytes(a->ggml_type) * 256 * a->rows, vb = b->row_bytes / block_bytes(b->ggml_type) * 256 * b->rows;
  return (va < vb ? va : vb) <= MMV_PAIR_VALUES;
}

int mmv_launch_pair_q81(int ta, int tb, const MmvArgs& a, const MmvArgs& b, int sm_count, int max_smem, cudaStream_t st);    // gsq_mmv_pair.cu
int mmv_launch_pair_xq81(int ta, int tb, const MmvArgs& a, const MmvArgs& b, int sm_count, int max_smem, cudaStream_t st);   // gsq_mmv_pair_x.cu

// Two products of the same activations in one launch (mmv_pair_kernel): 1..8 rows, both types at row counts that this kernel
// serves. x: block_q8_1 (x_dtype < 0), or X itself where both products would take that (mmv_raw_applies).
int mmv_pair_host(const gsq_weight* wa, const gsq_weight* wb, const void* x, int x_dtype, int64_t m, int64_t k, int64_t x_row_stride, int y_dtype,
                  int64_t y_row_stride, void* stream) {
  if (!mmv_pair_serves(wa, wb, m) || k <= 0 || k % 256 != 0 || k > INT32_MAX || !x || (y_dtype != GSQ_F32 && y_dtype != GSQ_F16 && y_dtype != GSQ_BF16) ||
      (x_dtype >= 0 && x_dtype != GSQ_F32 && x_dtype != GSQ_F16 && x_dtype != GSQ_BF16))
    return GSQ_ERR_UNSUPPORTED;
  for (const gsq_weight* w : {wa, wb}) {
    const int bs = block_bytes(w->ggml_type);
    if (!w->w || !w->y || w->rows < 1 || w->rows > INT32_MAX || bs == 0 || w->row_bytes != (k / 256) * bs || (x_dtype >= 0 && !mmv_raw_applies(w->ggml_type, w->packed, w->rows, m, k, 1)))
      return GSQ_ERR_UNSUPPORTED;
  }
  DeviceInfo di;
  const int rc = device_info(&di);
  if (rc != GSQ_OK) return rc;
  const MmvArgs a = mmv_args(wa->w, wa->row_bytes, wa->rows, x, m, k, wa->y, y_dtype, y_row_stride, nullptr, x_dtype, x_row_stride);
  const MmvArgs b = mmv_args(wb->w, wb->row_bytes, wb->rows, x, m, k, wb->y, y_dtype, y_row_stride, nullptr, x_dtype, x_row_stride);
  const int r = (x_dtype < 0 ? mmv_launch_pair_q81 : mmv_launch_pair_xq81)(wa->ggml_type, wb->ggml_type, a, b, di.sm_count, di.max_smem_optin,
                                                                          (cudaStream_t)stream);
  return r == MMV_DECLINED ? GSQ_ERR_UNSUPPORTED : r;
}

// Sticky flags of bounded waits that gave up: on a peer GPU, on a bulk copy.
int mmv_error_flags(int* peer, int* copy) {
  int p[4] = {0, 0, 0, 0}, c[4] = {0, 0, 0, 0};
  int rc = mmv_errors_q4k(&p[0], &c[0]);
  if (rc == GSQ_OK) rc = mmv_errors_iq4xs(&p[1], &c[1]);
  if (rc == GSQ_OK) rc = mmv_errors_iq3s(&p[2], &c[2]);
  if (rc == GSQ_OK) rc = mmv_errors_q6k(&p[3], &c[3]);
  *peer = p[0] | p[1] | p[2] | p[3];
  *copy = c[0] | c[1] | c[2] | c[3];
  return rc;
}

// The activations in the order of the staging area (quantize_rows_host): padded columns, bytes.
int mmv_rows_columns(int64_t m) {
  const int64_t ntl = (m + 7) / 8;
  return (int)(8 * (ntl == 5 ? 6 : ntl));
}
// Whether that order is the faster one: it is once a CTA's share of a column is some hundred bytes. Small weights are split
// over clusters of 8 and each copy is short (1024 x 2048 IQ3_S at 40 rows 7.8 us from blocks, 8.5 from rows); above 32 rows
// the scales of 48 columns and the more copies leave a gain only for large products of Q6_K (17408 x 5120 at 48 rows 55.4 ->
// 52.0; 5120 x 5120 24.9 -> 24.1, at 33 rows 24.1 -> 24.8) and the largest of IQ4_XS (17408 x 5120 at 33 and 48 rows 42.8 -> 41.2
// and 44.6 -> 40.9, 34816 x 5120 77.3 -> 75.8 and 79.7 -> 74.7, but 7168 x 5120 at 33 rows 24.9 -> 25.0; IQ3_S 43.7 -> 43.1, Q4_K
// 51.1 both).
bool mmv_rows_wins(int ggml_type, int64_t rows, int64_t m, int64_t k) {
  const int64_t least = m <= 32 ? 4 << 20 : ggml_type == GSQ_TYPE_Q6_K ? 16 << 20 : ggml_type == GSQ_TYPE_IQ4_XS ? 64 << 20 : INT64_MAX;
  return rows * k > least && k <= (1 << 24);
}
size_t mmv_rows_bytes(int ggml_type, int64_t m, int64_t k) {
  return (size_t)(m * k) + (size_t)(k / 32) * mmv_rows_columns(m) * (ggml_type == GSQ_TYPE_Q4_K ? 8 : 4);
}

}  // namespace gsq

extern "C" int gsq_peer_reduce_error_flag(int* flag) {
  int copy;
  return flag ? gsq::mmv_error_flags(flag, &copy) : GSQ_ERR_UNSUPPORTED;
}

extern "C" int gsq_debug_mmv_mode(int mode) {
  const int old = gsq::g_mmv_mode;
  gsq::g_mmv_mode = mode == 1 ? 1 : 0;
  return old;
}

extern "C" int gsq_debug_mmv_min_rows(int n) {
  const int old = gsq::g_mmv_min_rows;
  gsq::g_mmv_min_rows = n < 0 ? 0 : n;
  return old;
}

extern "C" int gsq_debug_mmv_max_rows(int n) {
  const int old = gsq::g_mmv_max_rows;
  gsq::g_mmv_max_rows = n > 48 ? 48 : n;
  return old;
}

extern "C" int gsq_mul_mat_vec_max_rows(int ggml_type, int packed) {
  return gsq::mmv_applies(ggml_type, packed, 16, gsq::g_mmv_max_rows) ? gsq::g_mmv_max_rows : 8;
}

extern "C" int gsq_debug_mmv_prefetch_first(int n) {
  const int old = gsq::g_mmv_pf_first;
  gsq::g_mmv_pf_first = n < 0 ? 0 : n > 64 ? 64 : n;
  return old;
}

extern "C" int gsq_debug_mmv_chunking(int mode) {
  const int old = gsq::g_mmv_aligned;
  gsq::g_mmv_aligned = (mode == 0 || mode == 1) ? mode : -1;
  return old;
}

extern "C" int gsq_debug_mmv_trace(int on) {
  const int old = gsq::g_mmv_trace;
  gsq::g_mmv_trace = on ? 1 : 0;
  return old;
}

extern "C" int gsq_debug_mmv_pdl(int on) {
  const int old = gsq::g_mmv_pdl;
  gsq::g_mmv_pdl = on < 0 ? 0 : on > 3 ? 3 : on;
  return old;
}

extern "C" int gsq_debug_mmv_profile(unsigned long long* stamps) {
  gsq::g_mmv_prof = stamps;
  return GSQ_OK;
}

extern "C" int gsq_debug_mmv_cluster_size(int cs) {
  const int old = gsq::g_mmv_cluster;
  gsq::g_mmv_cluster = (cs == 1 || cs == 2 || cs == 4 || cs == 8) ? cs : 0;
  return old;
}

extern "C" int gsq_linear_vec_pair(const gsq_weight* a, const gsq_weight* b, const void* x, int x_dtype, int64_t m, int64_t k, int64_t x_row_stride,
                                   int y_dtype, int64_t y_row_stride, void* stream) {
  if (!a || !b) return GSQ_ERR_UNSUPPORTED;
  return gsq::mmv_pair_host(a, b, x, x_dtype, m, k, x_row_stride, y_dtype, y_row_stride, stream);
}
extern "C" int gsq_linear_vec_pair_serves(const gsq_weight* a, const gsq_weight* b, int64_t m) { return a && b && gsq::mmv_pair_serves(a, b, m) ? 1 : 0; }
