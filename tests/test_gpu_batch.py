"""The kernel of up to 256 activation rows with exact integer slice sums and evenly cut work: every token-block size, ragged
row and token counts, tiles cut between CTAs at any superblock, against the reference kernels' arithmetic (fp32 scaling of
int32 slice sums, in float64)."""

import ctypes

import numpy as np
import pytest
import torch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, synth
from gsq_b200.quantization import iq3_pack
from oracle import blocks, product, q8_1

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = {"IQ3_S": 21, "IQ4_XS": 23, "Q4_K": 12}


@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("rows,k", [(16, 256), (144, 1024), (1040, 4608)])
@pytest.mark.parametrize("m", [1, 16, 17, 33, 49, 66, 96, 100, 113, 128, 129, 200, 256])
def test_batch_kernel(name, rows, k, m):
    t, packed = TYPES[name], name == "IQ3_S"
    raw = synth.make_weight(t, rows, k, 80 + rows)
    w = torch.from_numpy(raw).to(DEV)
    if packed:
        iq3_pack.pack_(w, t)
    xa = synth.make_activation(m, k, 81 + m)
    xa[0, :64] = 0.0
    xa[m - 1, 40] = 300.0
    x = synth.nudge_ties_torch(torch.from_numpy(xa).to(torch.bfloat16)).float()
    layout = q8_1.LAYOUT_DS4 if name == "Q4_K" else q8_1.LAYOUT_D4
    q, d, s = q8_1.quantize_mmq(x.numpy(), layout)
    dec = blocks.decode(raw, t)
    sums = product.block_sums(dec, q).astype(np.float64)
    scale = np.repeat(dec.d, 8, axis=1).astype(np.float64) * dec.isc
    if name == "Q4_K":   # half d and half sum x per block
        d, s = d.astype(np.float16), s.astype(np.float16)
    want = np.einsum("mns,ns,ms->mn", sums, scale, d.astype(np.float64), optimize=True)
    if name == "Q4_K":
        want -= s.astype(np.float64) @ (np.repeat(dec.dmin, 8, axis=1).astype(np.float64) * dec.imin).T
    lib = _cabi.lib
    old = lib.gsq_debug_gemm_variant(10)
    try:
        n = lib.gsq_linear_workspace_bytes(rows, m, k, t, int(packed))
        scratch = torch.full((n,), 0xFF, dtype=torch.uint8, device=DEV)
        y = torch.full((m, rows + 3), float("nan"), dtype=torch.float32, device=DEV)
        xd = x.to(DEV)
        rc = lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, int(packed), xd.data_ptr(), 0, m, k, k, y.data_ptr(), 0, rows + 3,
                            scratch.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, lib.gsq_strerror(rc)
        torch.cuda.synchronize()
    finally:
        lib.gsq_debug_gemm_variant(old)
    got = y[:, :rows].cpu().numpy()
    assert bool(torch.isnan(y[:, rows:]).all()) and np.isfinite(got).all()
    assert product.rel_err(got, want) <= 2e-6
    flag = ctypes.c_int(-1)
    assert lib.gsq_device_error_flag(ctypes.byref(flag)) == 0 and flag.value == 0
