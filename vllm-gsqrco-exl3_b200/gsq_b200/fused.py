"""The element-wise step in front of a quantised linear fused with its q8_1 quantiser (gsq_rmsnorm_quantize_q8_1,
gsq_silu_mul_quantize_q8_1): what a decoder layer does between two linears, in one launch each.

The reference's layers run vLLM's RMSNorm / SiluAndMul modules and quantise inside apply()
(plugin/vllm_gguf_plugin/quantization/linear.py:527-570 -> _quantize_x_q8_1, 251-268); these functions return the
block_q8_1 bytes that the vec ops take as their `x_q8` argument (torch.ops._C_gguf.lcpp_mul_mat_vec_* and
torch.ops.vllm._fused_mul_mat_gguf), plus, on request, the activations themselves for the other consumers.
"""

from __future__ import annotations

import torch

from . import _gsq_ops


def rmsnorm_quantize_q8_1(x: torch.Tensor, weight: torch.Tensor, eps: float, residual: torch.Tensor | None = None,
                          want_y: bool = False):
    """-> (x_q8, y or None). x [m, k]; weight [k] in x's dtype; residual: None, or [m, k] contiguous, updated in place to
    x + residual before the norm (vLLM's fused_add_rms_norm). x_q8: uint8 [m * k/32 * 36]."""
    return _gsq_ops.rmsnorm_quantize(x, weight, eps, residual, want_y)


def silu_mul_quantize_q8_1(gate_up: torch.Tensor, want_y: bool = False):
    """-> (x_q8, y or None). gate_up [m, 2 * inter], gate columns first; x_q8 of silu(gate) * up: uint8 [m * inter/32 * 36]."""
    return _gsq_ops.silu_mul_quantize(gate_up, want_y)
