"""Activations quantised in the small-batch product's own staging order: every column-group size and its padding, K split
unevenly over a cluster, strided X; bit for bit what the 128-value blocks give."""

import ctypes

import pytest
import torch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, synth
from gsq_b200.quantization import iq3_pack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("name,t", [("IQ3_S", 21), ("IQ4_XS", 23), ("Q4_K", 12), ("Q6_K", 14)])
@pytest.mark.parametrize("rows,k", [(8208, 768), (1040, 5120), (4112, 4352)])
@pytest.mark.parametrize("m", [5, 9, 16, 17, 24, 31, 32, 33, 41, 48])
def test_rows_equal_blocks(name, t, rows, k, m):
    lib, packed = _cabi.lib, name in ("IQ3_S", "Q6_K")
    w = torch.from_numpy(synth.make_weight(t, rows, k, 40)).to(DEV)
    if packed:
        iq3_pack.pack_(w, t)
    x = torch.from_numpy(synth.make_activation(m, k + 3, 41 + m)).to(DEV)
    x[0, :64] = 0.0
    st = torch.cuda.current_stream().cuda_stream
    out = []
    for n in (lib.gsq_linear_workspace_bytes(rows, m, k, t, int(packed)), lib.gsq_linear_scratch_bytes(rows, m, k, t, int(packed))):
        scratch = torch.full((n,), 0xFF, dtype=torch.uint8, device=DEV)
        y = torch.full((m, rows + 1), float("nan"), dtype=torch.float32, device=DEV)
        rc = lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, int(packed), x.data_ptr(), 0, m, k, k + 3, y.data_ptr(), 0, rows + 1,
                            scratch.data_ptr(), n, st)
        assert rc == 0, lib.gsq_strerror(rc)
        out.append(y)
    assert bool(torch.isfinite(out[0][:, :rows]).all()) and bool(torch.isnan(out[0][:, rows:]).all())
    assert torch.equal(out[0][:, :rows], out[1][:, :rows])
    flag = ctypes.c_int(-1)
    assert lib.gsq_device_error_flag(ctypes.byref(flag)) == 0 and flag.value == 0


@pytest.mark.parametrize("m", [33, 41, 48])
def test_rows_equal_blocks_on_large_weights_above_32_rows(m):
    """IQ4_XS weights of more than 64 M values."""
    test_rows_equal_blocks("IQ4_XS", 23, 13136, 5120, m)
