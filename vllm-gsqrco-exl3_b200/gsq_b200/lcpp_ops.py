"""torch.ops._C_gguf.lcpp_* -- the reference's C++ op schemas, served by libgsq.so.

Schemas are those of plugin/vllm_gguf_plugin/csrc/lcpp_shim.cu:973-983, verbatim. As there, every
op is registered for CUDA and for CPU: on CPU every guard runs and the call then ends in
"... must be CUDA tensors" (lcpp_shim.cu:997-1008), which is how guards are tested without a GPU.

What runs underneath an op name (lcpp_shim.cu:753-909 `run`):
  * the ops that read block_q8_1 activations (`x_q8` argument; vec_q, vec_iq3, vec_iq3_mma,
    vec_own, vec_iq3_mma_packed) -> gsq_quantize_q8_1 (unless x_q8 is given) + gsq_mul_mat_vec_q8,
    as many activation rows per launch as the kernel for the type takes (8 or 48);
  * the ops that quantise X themselves (mul_mat_q, mma_k, iq3_packed) -> gsq_linear, which picks
    the activation layout together with the kernel (small-batch tensor-core kernel, tcgen05 GEMM).
Implemented in native code (csrc/gsq_torch.cpp, module _gsq_ops). Output and scratch come from torch's caching
allocator on the current stream; the kernels write X's dtype directly, so no cast kernel follows.
"""

from __future__ import annotations

import ctypes as C
import os

import torch

from . import _cabi, _gsq_ops

_SCHEMAS = {
    "lcpp_mul_mat_vec_q": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "lcpp_mul_mat_q": "(Tensor W, Tensor X, int type, SymInt row) -> Tensor",
    "lcpp_mul_mat_vec_iq3": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "lcpp_mul_mat_vec_iq3_mma": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "lcpp_mul_mat_vec_own": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "lcpp_mul_mat_mma_k": "(Tensor W, Tensor X, int type, SymInt row) -> Tensor",
    "lcpp_mul_mat_vec_iq3_mma_packed": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "lcpp_mul_mat_iq3_packed": "(Tensor W, Tensor X, int type, SymInt row) -> Tensor",
    "lcpp_quantize_q8_1": "(Tensor X, int type, bool mmq, bool vendored) -> Tensor",
    # not in the reference: Q6_K repacked at load by this package (quantization/iq3_pack.py)
    "gsq_mul_mat_vec_q6k_packed": "(Tensor W, Tensor X, int type, SymInt row, Tensor? x_q8=None) -> Tensor",
    "gsq_mul_mat_q6k_packed": "(Tensor W, Tensor X, int type, SymInt row) -> Tensor",
    # nor this: a fused layer's runs of several types into one result (quantization/linear.py apply())
    "gsq_linear_runs": "(Tensor X, Tensor W, int[] runs, bool packed) -> Tensor",
}


class output_into:
    """with output_into(t): the next op call of this module on this thread writes its [rows of X, row] result into `t`
    (same shape and dtype as it would have returned, unit inner stride, any row stride) and returns `t`: the kernels take
    any row stride, so a tensor-parallel runtime can have a shard's result land in its slot of a collective's buffer
    instead of copying it there. A fused layer of several types is one call (gsq_linear_runs): `t` takes all its columns."""

    def __init__(self, t: torch.Tensor):
        self.t = t

    def __enter__(self):
        self._depth = _gsq_ops.push_output(self.t)
        return self.t

    def __exit__(self, *a):
        _gsq_ops.pop_output(self._depth)


class peer_reduce:
    """with peer_reduce(ctx): the next self-quantising op call of this module on this thread (lcpp_mul_mat_q,
    lcpp_mul_mat_mma_k, lcpp_mul_mat_iq3_packed, gsq_mul_mat_q6k_packed) is the product AND the sum of its result over the
    ranks of `ctx` (a _cabi.PeerReduce; tp.PeerAllReduce.fused()), one kernel (gsq_linear_allreduce). Raises if the shape
    is not one the small-batch kernel serves."""

    def __init__(self, ctx):
        self.ctx = ctx

    def __enter__(self):
        self._depth = _gsq_ops.push_peer(C.addressof(self.ctx))
        return self

    def __exit__(self, *a):
        _gsq_ops.pop_peer(self._depth)


def set_k_multiple(v: int) -> int:
    """K granularity the guards demand: 512 as in the reference (MATRIX_ROW_PADDING); the tensor-parallel helpers lower
    it to 256 for K-sharded layers (gsq_b200.tp.relaxed_k). Returns the previous value."""
    return _gsq_ops.set_k_multiple(int(v))


PREFILL_ROUNDED, PREFILL_SPLIT, PREFILL_INTEGER = 0, 1, 2


def set_prefill_precision(mode: int) -> int:
    """How the prefill products of repacked IQ3_S, IQ4_XS and Q4_K are formed (gsq_prefill_precision): PREFILL_ROUNDED
    (default; within about 4e-4 of a row's norm of the reference kernels' result), PREFILL_SPLIT (IQ3_S: about 1e-6),
    PREFILL_INTEGER (the reference's exact integer slice sums, which Q6_K keeps in every mode). Returns the previous mode. The environment variable GSQ_PREFILL_PRECISION
    (rounded / split / integer) sets it at import."""
    return int(_cabi.lib.gsq_prefill_precision(int(mode)))


def _make_fake(name):
    if name == "lcpp_quantize_q8_1":
        return lambda X, type, mmq, vendored: X.new_empty(
            (X.shape[0] * X.shape[1] // 128 * 144 if mmq else X.shape[0] * X.shape[1] // 32 * 36,), dtype=torch.uint8)
    if name == "gsq_linear_runs":
        return lambda X, W, runs, packed: X.new_empty((X.shape[0], sum(runs[1::4])))
    if "x_q8" in _SCHEMAS[name]:
        return lambda W, X, type, row, x_q8=None: X.new_empty((X.shape[0], row))
    return lambda W, X, type, row: X.new_empty((X.shape[0], row))


_LIBRARY = None
registered: list[str] = []


def register() -> list[str]:
    """Define and implement the ops once per process. If another extension has already defined an op of
    this name in `_C_gguf` (the reference's own .so), that definition is left alone and the name is
    not in the returned list."""
    global _LIBRARY
    if _LIBRARY is not None:
        return registered
    want = os.environ.get("GSQ_PREFILL_PRECISION", "").strip().lower()
    if want:
        modes = {"rounded": PREFILL_ROUNDED, "split": PREFILL_SPLIT, "integer": PREFILL_INTEGER}
        if want not in modes:
            raise ValueError(f"GSQ_PREFILL_PRECISION={want!r}: expected one of {sorted(modes)}")
        set_prefill_precision(modes[want])
    _LIBRARY = torch.library.Library("_C_gguf", "FRAGMENT")
    for name, schema in _SCHEMAS.items():
        try:
            _LIBRARY.define(name + schema)
        except RuntimeError:
            continue
        _gsq_ops.implement(name)
        _LIBRARY._register_fake(name, _make_fake(name))
        registered.append(name)
    return registered
