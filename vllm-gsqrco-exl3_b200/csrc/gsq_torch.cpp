// Host path of the quantised linear in native code: the implementations of torch.ops._C_gguf.*, of
// torch.ops.vllm._fused_mul_mat_gguf, and the same calls as plain Python functions (module gsq_b200._gsq_ops).
//
// What bounds it: a decode-sized product takes 8 to 20 us on the GPU, and with the ops implemented in Python (dispatcher
// -> Python -> ctypes, guards filled field by field) one call took 42 us of host time, 126 us for a fused layer of two
// runs: the GPU idled between calls. Here a call is one dispatch, the guards on a stack structure, one or two
// caching-allocator calls and the launches.
//
// Everything the ops mean is unchanged: the op table, guards (gsq_check_inputs) and messages, the routing table
// (gsq_b200/quantization/linear.py `_lcpp_op`, restated in route() below and compared with it point by point in
// tests/test_host_ops.py), buffers from torch's caching allocator on the current stream.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>
#include <torch/library.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/gsq.h"

namespace {

using at::Tensor;

enum Op {
  VEC_Q, MUL_MAT_Q, VEC_IQ3, VEC_IQ3_MMA, VEC_OWN, MMA_K, VEC_IQ3_MMA_PACKED, IQ3_PACKED, VEC_Q6K_PACKED, Q6K_PACKED, N_OPS
};
// vec: reads block_q8_1 activations (its x_q8 argument); the others quantise X themselves
struct Spec {
  const char* name;
  bool vec, packed, need_iq3, need_q4k_own, need_mma_k, is_mmq, need_q6k;
  int max_rows;
};
const Spec kSpec[N_OPS] = {
    {"lcpp_mul_mat_vec_q", true, false, false, false, false, false, false, 8},
    {"lcpp_mul_mat_q", false, false, false, false, false, true, false, 0},
    {"lcpp_mul_mat_vec_iq3", true, false, true, false, false, false, false, 8},
    {"lcpp_mul_mat_vec_iq3_mma", true, false, true, false, false, false, false, 8},
    {"lcpp_mul_mat_vec_own", true, false, false, true, false, false, false, 8},
    {"lcpp_mul_mat_mma_k", false, false, false, false, true, false, false, 64},
    {"lcpp_mul_mat_vec_iq3_mma_packed", true, true, true, false, false, false, false, 32},
    {"lcpp_mul_mat_iq3_packed", false, true, true, false, false, false, false, 0},
    {"gsq_mul_mat_vec_q6k_packed", true, true, false, false, false, false, true, 8},
    {"gsq_mul_mat_q6k_packed", false, true, false, false, false, false, true, 0},
};

constexpr int Q2_K = 10, Q4_K = 12, Q6_K = 14, IQ2_XXS = 16, IQ2_XS = 17, IQ3_XXS = 18, IQ3_S = 21, IQ2_S = 22, IQ4_XS = 23, IQ1_M = 29;

struct Switches {
  int k_multiple = 512;
  bool enabled = true, mma_k = true, iq3_tiled = true, iq1m_mmvq = true;
};
Switches g_sw;

// what the next op call of this thread writes into / sums with (lcpp_ops.output_into, lcpp_ops.peer_reduce)
thread_local std::vector<Tensor> t_outputs;
thread_local std::vector<gsq_peer_reduce> t_peers;

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? GSQ_F32 : t == at::kHalf ? GSQ_F16 : t == at::kBFloat16 ? GSQ_BF16 : GSQ_DTYPE_OTHER;
}

void check(int status, const char* what) {
  if (status == GSQ_OK) return;
  std::string msg = std::string(what) + ": " + gsq_strerror(status);
  if (status == GSQ_ERR_CUDA) msg += " (cudaError " + std::to_string(gsq_last_cuda_error()) + ")";
  TORCH_CHECK(false, msg);
}

bool quant_type(int64_t t) {
  switch (t) {
    case Q2_K: case Q4_K: case Q6_K: case IQ2_XXS: case IQ2_XS: case IQ3_XXS: case IQ3_S: case IQ2_S: case IQ4_XS: case IQ1_M: return true;
    default: return false;
  }
}
bool packable(int64_t t) { return t == IQ3_S || t == Q6_K; }

// Op for n activation rows times a `type` weight of `rows` x `k`, -1 if there is none: linear.py `_lcpp_op`, with the two
// ops of repacked Q6_K in place of the table's names as `_fused_mul_mat_gguf` puts them.
int route(int64_t n, int64_t type, int64_t rows, int64_t k, bool packed) {
  const bool iq3 = type == IQ3_S || type == IQ3_XXS;
  if (iq3 && packed) return n <= 8 || !g_sw.iq3_tiled ? VEC_IQ3_MMA_PACKED : IQ3_PACKED;
  if (type == IQ1_M) return n <= 8 || (n <= 32 && g_sw.iq1m_mmvq) ? VEC_Q : -1;
  int op = n >= 8 ? MUL_MAT_Q : VEC_Q;
  if (n <= 8 && iq3) {
    op = n < 6 ? VEC_IQ3 : VEC_IQ3_MMA;
  } else if (n <= 8 && rows > 2048 && n >= (type == Q4_K ? 3 : type == IQ2_S ? 1 : 9)) {
    op = VEC_OWN;
  } else if (g_sw.mma_k && (type == Q4_K || type == IQ4_XS || type == IQ2_S) && n >= 9 && n <= 32 && rows > 2048 &&
             (type != IQ4_XS || n <= 16 || rows * k >= 12288ll * 5120)) {
    op = MMA_K;
  }
  if (packed && type == Q6_K) op = op == VEC_Q ? VEC_Q6K_PACKED : Q6K_PACKED;
  return op;
}

// One weight: bytes, shape and strides as the guards want them (a tensor, or rows of a fused layer's buffer).
struct Weight {
  const uint8_t* data;
  int64_t dim, size0, size1, stride0, stride1;
  bool is_uint8, is_cuda;
  c10::Device device;
};
Weight weight_of(const Tensor& w) {
  const bool two = w.dim() == 2;
  return {w.numel() ? (const uint8_t*)w.const_data_ptr() : nullptr, w.dim(), two ? w.size(0) : 0, two ? w.size(1) : 0,
          two ? w.stride(0) : 0, two ? w.stride(1) : 0, w.scalar_type() == at::kByte, w.is_cuda(), w.device()};
}

int64_t guard(const Spec& s, const Weight& w, const Tensor& x, int64_t type, int64_t row) {
  TORCH_CHECK(!s.need_q6k || type == Q6_K, s.name, ": Q6_K only, got type ", type);
  gsq_guard_args a = {};
  a.op = s.name;
  a.w_dim = (int)w.dim;
  a.w_is_uint8 = w.is_uint8;
  a.w_size0 = w.size0;
  a.w_size1 = w.size1;
  a.w_stride0 = w.stride0;
  a.w_stride1 = w.stride1;
  a.w_addr = (uint64_t)(uintptr_t)w.data;
  a.x_dim = (int)x.dim();
  a.x_dtype = dtype_code(x.scalar_type());
  if (x.dim() == 2) {
    a.x_size0 = x.size(0);
    a.x_size1 = x.size(1);
    a.x_stride0 = x.stride(0);
    a.x_stride1 = x.stride(1);
  }
  a.row = row;
  a.max_rows = s.max_rows;
  a.ggml_type = (int)type;
  a.need_iq3 = s.need_iq3;
  a.need_q4k_own = s.need_q4k_own;
  a.need_mma_k = s.need_mma_k;
  a.is_mmq = s.is_mmq;
  a.packed = s.packed;
  a.k_multiple = g_sw.k_multiple;
  a.w_is_cuda = w.is_cuda;
  a.x_is_cuda = x.is_cuda();
  a.same_device = w.device == x.device();
  int64_t k = 0;
  char msg[512];
  TORCH_CHECK(gsq_check_inputs(&a, &k, msg, sizeof(msg)) == GSQ_OK, msg);
  return k;
}

Tensor bytes(int64_t n, const Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }
int64_t row_stride(const Tensor& x, int64_t k) { return x.size(0) == 1 ? k : x.stride(0); }

Tensor quantize_blocks(const Tensor& x, int64_t k, void* stream) {
  Tensor q = bytes(x.size(0) * k / 32 * 36, x);
  check(gsq_quantize_q8_1(x.const_data_ptr(), dtype_code(x.scalar_type()), x.size(0), k, row_stride(x, k), q.mutable_data_ptr(), stream),
        "gsq_quantize_q8_1");
  return q;
}

void check_x_q8(const Spec& s, const Tensor& q, const Tensor& x, int64_t k) {
  const int64_t need = x.size(0) * k / 32 * 36;
  TORCH_CHECK(q.scalar_type() == at::kByte && q.dim() == 1 && q.stride(0) == 1 && q.numel() >= need, s.name,
              ": x_q8 must be contiguous uint8 with at least ", need, " bytes");
  TORCH_CHECK((uintptr_t)q.const_data_ptr() % 16 == 0, s.name, ": x_q8 must be 16-byte aligned");
  TORCH_CHECK(q.is_cuda() && q.device() == x.device(), s.name, ": x_q8 must be on X's device");
}

Tensor result(int64_t n, int64_t row, const Tensor& x) {
  if (!t_outputs.empty()) {
    Tensor y = std::move(t_outputs.back());
    t_outputs.pop_back();
    TORCH_CHECK(y.dim() == 2 && y.size(0) == n && y.size(1) == row && y.scalar_type() == x.scalar_type() && y.device() == x.device() &&
                    y.stride(1) == 1,
                "output_into: the tensor does not match the result's shape, dtype, device or inner stride");
    return y;
  }
  return at::empty({n, row}, x.options());
}

// Scratch of gsq_linear: what its fastest kernels want, or, where the allocator cannot give that, the least it runs in
// (expanded weights take 2 to 4 bytes a value: 566 MB for a 6-bit head at 128 rows, which runs in 0.7 MB as well).
Tensor linear_scratch(int64_t row, int64_t n, int64_t k, int type, bool packed, const Tensor& x) {
  const size_t most = gsq_linear_workspace_bytes(row, n, k, type, packed);
  try {
    return bytes(std::max<int64_t>((int64_t)most, 1), x);
  } catch (const c10::OutOfMemoryError&) {
    const size_t least = gsq_linear_scratch_bytes(row, n, k, type, packed);
    if (least >= most) throw;
    return bytes((int64_t)least, x);
  }
}

// Rows [i0, i0 + n) of x times w into y (row 0 of y = row i0 of x, row stride ldy) by one op; x, w guarded, k known, the
// device current. x_q8: block_q8_1 of all of x, made here if the op reads it and there is none yet.
void product(const Spec& s, const Weight& w, const Tensor& x, int64_t i0, int64_t n, int64_t type, int64_t row, int64_t k, Tensor& x_q8,
             char* y, int64_t ldy, void* stream) {
  const int dt = dtype_code(x.scalar_type());
  const int64_t es = x.element_size();
  if (s.vec) {
    if (!x_q8.defined() && n <= 8) {
      // quantised inside the product kernel where that is the faster way
      const int64_t xs = row_stride(x, k);
      const int rc = gsq_linear_vec(w.data, w.size1, row, (int)type, s.packed, (const char*)x.const_data_ptr() + i0 * xs * es, dt, n, k, xs, y,
                                    dt, ldy, stream);
      if (rc != GSQ_ERR_UNSUPPORTED) return check(rc, "gsq_linear_vec");
    }
    if (!x_q8.defined()) x_q8 = quantize_blocks(x, k, stream);
    const int64_t per_row = k / 32 * 36, step = gsq_mul_mat_vec_max_rows((int)type, s.packed);
    for (int64_t i = 0; i < n; i += step) {
      check(gsq_mul_mat_vec_q8(w.data, w.size1, row, (int)type, s.packed, (const char*)x_q8.const_data_ptr() + (i0 + i) * per_row,
                               std::min(step, n - i), k, y + i * ldy * es, dt, ldy, stream),
            "gsq_mul_mat_vec_q8");
    }
    return;
  }
  Tensor scratch = linear_scratch(row, n, k, (int)type, s.packed, x);
  const size_t have = (size_t)scratch.numel();
  const int64_t xs = row_stride(x, k);
  const char* xp = (const char*)x.const_data_ptr() + i0 * xs * es;
  if (!t_peers.empty()) {
    const gsq_peer_reduce pr = t_peers.back();
    t_peers.pop_back();
    check(gsq_linear_allreduce(w.data, w.size1, row, (int)type, s.packed, xp, dt, n, k, xs, y, dt, ldy, scratch.mutable_data_ptr(), have,
                               &pr, stream),
          "gsq_linear_allreduce");
    return;
  }
  check(gsq_linear(w.data, w.size1, row, (int)type, s.packed, xp, dt, n, k, xs, y, dt, ldy, scratch.mutable_data_ptr(), have, stream),
        "gsq_linear");
}

Tensor run_op(int op, const Tensor& w, const Tensor& x, int64_t type, int64_t row, const std::optional<Tensor>& x_q8) {
  const Spec& s = kSpec[op];
  const Weight wt = weight_of(w);
  const int64_t k = guard(s, wt, x, type, row), n = x.size(0);
  Tensor q = x_q8.value_or(Tensor());
  if (q.defined()) check_x_q8(s, q, x, k);
  if (n == 0) return at::empty({0, row}, x.options());
  const c10::cuda::CUDAGuard dev(x.device());
  Tensor y = result(n, row, x);
  product(s, wt, x, 0, n, type, row, k, q, (char*)y.mutable_data_ptr(), y.stride(0), c10::cuda::getCurrentCUDAStream().stream());
  return y;
}

// op of a product of apply(), with the errors `_fused_mul_mat_gguf` raises; `packed` in: the layer's flag, out: the run's
int op_for(int64_t n, int64_t type, int64_t rows, int64_t k, bool& packed) {
  TORCH_CHECK(g_sw.enabled, "VLLM_GGUF_LCPP=0: this package only implements that route and has no other path");
  TORCH_CHECK_NOT_IMPLEMENTED(quant_type(type), "Unsupported GGUF quantization type: ", type);
  packed = packed && packable(type);
  const int op = route(n, type, rows, k, packed);
  TORCH_CHECK_NOT_IMPLEMENTED(op >= 0, "no kernel for ggml type ", type, " at ", n, " activation rows");
  return op;
}

// One run of a product: guarded, then in calls of as many rows as its op takes (more than one call only with
// VLLM_GGUF_IQ3_TILED=0 or for IQ1_M above 8 rows).
void product_of_run(int op, const Weight& w, const Tensor& x, int64_t type, int64_t rows, Tensor& q, char* y, int64_t ldy, void* stream) {
  const Spec& s = kSpec[op];
  const int64_t n = x.size(0), per_call = !s.vec ? n : op == VEC_IQ3_MMA_PACKED ? 32 : 8;
  const int64_t k = guard(s, w, n > per_call ? x.narrow(0, 0, per_call) : x, type, rows);
  if (q.defined() && s.vec) check_x_q8(s, q, x, k);
  for (int64_t i = 0; i < n; i += per_call)
    product(s, w, x, i, std::min(per_call, n - i), type, rows, k, q, y + i * ldy * x.element_size(), ldy, stream);
}

// Two runs' products in one launch, side by side in y, where both ops read block_q8_1: to 7 rows (at 8 the routing table gives one of
// every pair's types an op on 128-value blocks), the types in the order of mmv_pair_types. False: no such kernel.
bool product_of_two(const Weight& wa, int64_t ta, const Weight& wb, int64_t tb, const Tensor& x, bool packed, Tensor& q, char* y, int64_t ldy,
                    void* stream) {
  const int64_t n = x.size(0);
  gsq_weight a = {wa.data, wa.size1, wa.size0, (int)ta, packed && packable(ta), y}, b = {wb.data, wb.size1, wb.size0, (int)tb, packed && packable(tb), y + wa.size0 * x.element_size()};
  if (!gsq_linear_vec_pair_serves(&a, &b, n) || dtype_code(x.scalar_type()) == GSQ_DTYPE_OTHER) return false;
  bool pa = packed, pb = packed;
  const int oa = op_for(n, ta, wa.size0, x.size(1), pa), ob = op_for(n, tb, wb.size0, x.size(1), pb);
  if (!kSpec[oa].vec || !kSpec[ob].vec) return false;
  const int64_t k = guard(kSpec[oa], wa, x, ta, wa.size0);
  guard(kSpec[ob], wb, x, tb, wb.size0);
  a.packed = kSpec[oa].packed;
  b.packed = kSpec[ob].packed;
  const int dt = dtype_code(x.scalar_type());
  int rc = GSQ_ERR_UNSUPPORTED;
  if (!q.defined()) rc = gsq_linear_vec_pair(&a, &b, x.const_data_ptr(), dt, n, k, row_stride(x, k), dt, ldy, stream);
  if (rc == GSQ_ERR_UNSUPPORTED) {
    if (!q.defined()) q = quantize_blocks(x, k, stream);
    rc = gsq_linear_vec_pair(&a, &b, q.const_data_ptr(), -1, n, k, 0, dt, ldy, stream);
  }
  if (rc == GSQ_ERR_UNSUPPORTED) return false;
  check(rc, "gsq_linear_vec_pair");
  return true;
}

Tensor unquantized(const Tensor& x, const Tensor& w) {
  if (x.size(0) <= 8 && w.size(0) <= 128) return at::bmm(x.unsqueeze(1), w.t().expand({x.size(0), -1, -1})).squeeze(1);
  return at::linear(x, w);
}

Tensor linear(const Tensor& x, const Tensor& w, int64_t type, const std::optional<Tensor>& x_q8, bool packed) {
  const int64_t n = x.size(0), rows = w.size(0);
  if (n == 0) return at::empty({0, rows}, x.options());
  if (type == 0 || type == 1 || type == 30) return unquantized(x, w);   // F32, F16, BF16
  TORCH_CHECK(x.dim() == 2, "X must be 2-D");
  const int op = op_for(n, type, rows, x.size(1), packed);
  const c10::cuda::OptionalCUDAGuard dev(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  Tensor q = x_q8.value_or(Tensor());
  const Weight wt = weight_of(w);
  if (!x.is_cuda()) guard(kSpec[op], wt, x, type, rows);   // ends in its message: there is nothing to run on
  Tensor y = result(n, rows, x);
  product_of_run(op, wt, x, type, rows, q, (char*)y.mutable_data_ptr(), y.stride(0), c10::cuda::getCurrentCUDAStream().stream());
  return y;
}

// A fused layer: `w` holds runs of adjacent same-type shards (weight rows `start` on, `rows` of them, stored as
// contiguous rows of `row_bytes` from there), `runs` = start, rows, row_bytes, type of each. All runs write their columns
// of one result, and share one block_q8_1 of x where their ops read that.
Tensor linear_runs(const Tensor& x, const Tensor& w, at::IntArrayRef runs, bool packed) {
  TORCH_CHECK(runs.size() % 4 == 0 && x.dim() == 2 && w.dim() == 2 && w.is_contiguous(), "gsq_linear_runs: bad arguments");
  int64_t total = 0, esz = w.element_size(), bytes_all = w.numel() * esz;
  bool plain = false;
  for (size_t i = 0; i < runs.size(); i += 4) {
    TORCH_CHECK(runs[i] >= 0 && runs[i + 1] > 0 && (runs[i] * w.size(1) + runs[i + 1] * runs[i + 2]) * esz <= bytes_all,
                "gsq_linear_runs: a run lies outside the weight");
    total += runs[i + 1];
    plain |= runs[i + 3] == 0 || runs[i + 3] == 1 || runs[i + 3] == 30;
  }
  const int64_t n = x.size(0);
  TORCH_CHECK(!plain, "gsq_linear_runs: quantised runs only");
  if (n == 0) return at::empty({0, total}, x.options());
  const c10::cuda::OptionalCUDAGuard dev(x.is_cuda() ? std::optional<c10::Device>(x.device()) : std::nullopt);
  Tensor y, q;
  int64_t col = 0;
  auto weight = [&](size_t i) {
    return Weight{(const uint8_t*)w.const_data_ptr() + runs[i] * w.size(1), 2, runs[i + 1], runs[i + 2], runs[i + 2], 1,
                  w.scalar_type() == at::kByte, w.is_cuda(), w.device()};
  };
  for (size_t i = 0; i < runs.size(); i += 4) {
    const int64_t rows = runs[i + 1], type = runs[i + 3];
    const Weight wt = weight(i);
    if (i + 4 < runs.size() && n <= 8 && x.is_cuda() && t_peers.empty()) {
      // two runs in one launch, where there is such a kernel
      const Weight wn = weight(i + 4);
      if (!y.defined()) y = result(n, total, x);
      if (product_of_two(wt, type, wn, runs[i + 7], x, packed, q, (char*)y.mutable_data_ptr() + col * x.element_size(), y.stride(0),
                         c10::cuda::getCurrentCUDAStream().stream())) {
        col += rows + runs[i + 5];
        i += 4;
        continue;
      }
    }
    bool pk = packed;
    const int op = op_for(n, type, rows, x.size(1), pk);
    if (!x.is_cuda()) guard(kSpec[op], wt, x, type, rows);
    if (!y.defined()) y = result(n, total, x);
    product_of_run(op, wt, x, type, rows, q, (char*)y.mutable_data_ptr() + col * x.element_size(), y.stride(0),
                   c10::cuda::getCurrentCUDAStream().stream());
    col += rows;
  }
  return y;
}

Tensor quantize_q8_1(const Tensor& x, int64_t type, bool mmq, bool vendored) {
  const int dt = dtype_code(x.scalar_type());
  TORCH_CHECK(gsq_type_block_bytes((int)type) > 0 && x.is_cuda() && x.dim() == 2 && x.stride(1) == 1 && x.size(1) % g_sw.k_multiple == 0 &&
                  dt != GSQ_DTYPE_OTHER,
              "lcpp_quantize_q8_1: bad arguments");
  const int64_t n = x.size(0), k = x.size(1);
  TORCH_CHECK(!vendored || (dt == GSQ_F32 && row_stride(x, k) % 4 == 0), "vendored: fp32 X");
  const c10::cuda::CUDAGuard dev(x.device());
  void* st = c10::cuda::getCurrentCUDAStream().stream();
  if (!mmq) return n ? quantize_blocks(x, k, st) : bytes(0, x);
  Tensor out = bytes(n * k / 128 * 144, x);
  if (n)
    check(gsq_quantize_q8_1_mmq(x.const_data_ptr(), dt, n, k, row_stride(x, k), gsq_q8_layout_for_type((int)type), out.mutable_data_ptr(), st),
          "gsq_quantize_q8_1_mmq");
  return out;
}

Tensor quantize_x_q8_1(const Tensor& x, at::IntArrayRef types, at::IntArrayRef rows, bool packed) {
  const int64_t n = x.size(0), k = x.size(1);
  for (size_t i = 0; n && i < types.size() && i < rows.size(); ++i) {
    if (!quant_type(types[i])) continue;
    // (the table's own op decides, before the substitution for repacked Q6_K)
    const int op = route(n, types[i], rows[i], k, packed && types[i] != Q6_K);
    if (op >= 0 && kSpec[op].vec) return quantize_q8_1(x, types[i], false, false);
  }
  return bytes(n * k / 32 * 36, x);
}

// ---- the fused front ends (gsq_b200.fused)

std::tuple<Tensor, std::optional<Tensor>> rmsnorm_quantize(const Tensor& x, const Tensor& weight, double eps, const std::optional<Tensor>& residual,
                                                           bool want_y) {
  const int dt = dtype_code(x.scalar_type());
  TORCH_CHECK(x.is_cuda() && x.dim() == 2 && x.stride(1) == 1 && dt != GSQ_DTYPE_OTHER && x.size(1) % 32 == 0,
              "rmsnorm_quantize_q8_1: x must be a CUDA [m, k] tensor, unit inner stride, k % 32 == 0");
  const int64_t m = x.size(0), k = x.size(1);
  TORCH_CHECK(weight.dim() == 1 && weight.size(0) == k && weight.scalar_type() == x.scalar_type() && weight.device() == x.device() &&
                  weight.is_contiguous(),
              "rmsnorm_quantize_q8_1: weight must be [k] in x's dtype on x's device");
  TORCH_CHECK(!residual || (residual->sizes() == x.sizes() && residual->scalar_type() == x.scalar_type() && residual->is_contiguous() &&
                            residual->device() == x.device()),
              "rmsnorm_quantize_q8_1: residual must be contiguous and match x");
  const c10::cuda::CUDAGuard dev(x.device());
  Tensor q = bytes(m * k / 32 * 36, x);
  std::optional<Tensor> y;
  if (want_y) y = at::empty({m, k}, x.options());
  if (m)
    check(gsq_rmsnorm_quantize_q8_1(x.const_data_ptr(), dt, m, k, row_stride(x, k), residual ? residual->mutable_data_ptr() : nullptr,
                                    weight.const_data_ptr(), (float)eps, q.mutable_data_ptr(), y ? y->mutable_data_ptr() : nullptr,
                                    c10::cuda::getCurrentCUDAStream().stream()),
          "gsq_rmsnorm_quantize_q8_1");
  return {q, y};
}

std::tuple<Tensor, std::optional<Tensor>> silu_mul_quantize(const Tensor& gate_up, bool want_y) {
  const int dt = dtype_code(gate_up.scalar_type());
  TORCH_CHECK(gate_up.is_cuda() && gate_up.dim() == 2 && gate_up.stride(1) == 1 && dt != GSQ_DTYPE_OTHER && gate_up.size(1) % 64 == 0,
              "silu_mul_quantize_q8_1: gate_up must be a CUDA [m, 2 * inter] tensor, unit inner stride, inter % 32 == 0");
  const int64_t m = gate_up.size(0), inter = gate_up.size(1) / 2;
  const c10::cuda::CUDAGuard dev(gate_up.device());
  Tensor q = bytes(m * inter / 32 * 36, gate_up);
  std::optional<Tensor> y;
  if (want_y) y = at::empty({m, inter}, gate_up.options());
  if (m)
    check(gsq_silu_mul_quantize_q8_1(gate_up.const_data_ptr(), dt, m, inter, row_stride(gate_up, 2 * inter), q.mutable_data_ptr(),
                                     y ? y->mutable_data_ptr() : nullptr, c10::cuda::getCurrentCUDAStream().stream()),
          "gsq_silu_mul_quantize_q8_1");
  return {q, y};
}

// ---- registration. The ops are defined in Python (which leaves names alone that another extension has defined); the
// implementations are added here, one library object per (namespace, key) kept for the process's life.

template <int OP>
Tensor op_vec(const Tensor& w, const Tensor& x, int64_t type, int64_t row, const std::optional<Tensor>& x_q8) {
  return run_op(OP, w, x, type, row, x_q8);
}
template <int OP>
Tensor op_self(const Tensor& w, const Tensor& x, int64_t type, int64_t row) {
  return run_op(OP, w, x, type, row, std::nullopt);
}

torch::Library& library(const char* ns, c10::DispatchKey key) {
  static std::vector<std::pair<std::pair<std::string, c10::DispatchKey>, std::unique_ptr<torch::Library>>> libs;
  for (auto& l : libs)
    if (l.first.first == ns && l.first.second == key) return *l.second;
  libs.emplace_back(std::make_pair(std::string(ns), key), std::make_unique<torch::Library>(torch::Library::IMPL, ns, key, __FILE__, __LINE__));
  return *libs.back().second;
}

void implement(const std::string& name) {
  for (auto key : {c10::DispatchKey::CUDA, c10::DispatchKey::CPU}) {
    auto& l = library("_C_gguf", key);
    const char* n = name.c_str();
    if (name == kSpec[VEC_Q].name) l.impl(n, &op_vec<VEC_Q>);
    else if (name == kSpec[MUL_MAT_Q].name) l.impl(n, &op_self<MUL_MAT_Q>);
    else if (name == kSpec[VEC_IQ3].name) l.impl(n, &op_vec<VEC_IQ3>);
    else if (name == kSpec[VEC_IQ3_MMA].name) l.impl(n, &op_vec<VEC_IQ3_MMA>);
    else if (name == kSpec[VEC_OWN].name) l.impl(n, &op_vec<VEC_OWN>);
    else if (name == kSpec[MMA_K].name) l.impl(n, &op_self<MMA_K>);
    else if (name == kSpec[VEC_IQ3_MMA_PACKED].name) l.impl(n, &op_vec<VEC_IQ3_MMA_PACKED>);
    else if (name == kSpec[IQ3_PACKED].name) l.impl(n, &op_self<IQ3_PACKED>);
    else if (name == kSpec[VEC_Q6K_PACKED].name) l.impl(n, &op_vec<VEC_Q6K_PACKED>);
    else if (name == kSpec[Q6K_PACKED].name) l.impl(n, &op_self<Q6K_PACKED>);
    else if (name == "lcpp_quantize_q8_1") l.impl(n, &quantize_q8_1);
    else if (name == "gsq_linear_runs") l.impl(n, &linear_runs);
    else TORCH_CHECK(false, "no implementation of ", name);
  }
}

void implement_vllm(const std::string& name) {
  auto& l = library("vllm", c10::DispatchKey::CUDA);
  if (name == "_fused_mul_mat_gguf") l.impl(name.c_str(), &linear);
  else if (name == "_quantize_x_q8_1") l.impl(name.c_str(), &quantize_x_q8_1);
  else TORCH_CHECK(false, "no implementation of ", name);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("implement", &implement);
  m.def("implement_vllm", &implement_vllm);
  // The calls that launch let go of the interpreter, as the custom ops do: the allocator may wait for the driver in them.
  using free_interpreter = pybind11::call_guard<pybind11::gil_scoped_release>;
  m.def("linear", &linear, free_interpreter());
  m.def("linear_runs", [](const Tensor& x, const Tensor& w, const std::vector<int64_t>& runs, bool packed) { return linear_runs(x, w, runs, packed); },
        free_interpreter());
  m.def("rmsnorm_quantize", &rmsnorm_quantize, free_interpreter());
  m.def("silu_mul_quantize", &silu_mul_quantize, free_interpreter());
  m.def("route", [](int64_t n, int64_t type, int64_t rows, int64_t k, bool packed) -> std::optional<std::string> {
    const int op = route(n, type, rows, k, packed);
    return op < 0 ? std::nullopt : std::optional<std::string>(kSpec[op].name);
  });
  m.def("set_k_multiple", [](int v) { return std::exchange(g_sw.k_multiple, v); });
  m.def("set_switches", [](bool enabled, bool mma_k, bool iq3_tiled, bool iq1m_mmvq) {
    g_sw.enabled = enabled;
    g_sw.mma_k = mma_k;
    g_sw.iq3_tiled = iq3_tiled;
    g_sw.iq1m_mmvq = iq1m_mmvq;
  });
  m.def("push_output", [](const Tensor& t) { t_outputs.push_back(t); return (int64_t)t_outputs.size(); });
  m.def("pop_output", [](int64_t depth) { if ((int64_t)t_outputs.size() >= depth) t_outputs.resize(depth - 1); });
  m.def("push_peer", [](uintptr_t p) { t_peers.push_back(*(const gsq_peer_reduce*)p); return (int64_t)t_peers.size(); });
  m.def("pop_peer", [](int64_t depth) { if ((int64_t)t_peers.size() >= depth) t_peers.resize(depth - 1); });
}
