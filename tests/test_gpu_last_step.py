"""The last step of the small-batch product at 1 to 16 rows, where a thread's group of four columns comes from its number: every
share of the threads, partial groups, fewer and more rows of a CTA than a share has threads, rows of Y past the weight's."""

import numpy as np
import pytest
import torch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, synth
from gsq_b200.quantization import iq3_pack
from oracle import blocks, product, q8_1

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = {"IQ3_S": 21, "IQ4_XS": 23, "Q4_K": 12, "Q6_K": 14}


@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("rows,k", [(16, 256), (2384, 768), (80016, 256)])
def test_every_share_of_the_threads(name, rows, k):
    t, packed, lib = TYPES[name], name in ("IQ3_S", "Q6_K"), _cabi.lib
    rows -= 0 if packed else 13   # (repacked weights are whole 16-row records)
    raw = synth.make_weight(t, rows, k, 60 + k)
    dec = blocks.decode(raw, t)
    w = torch.from_numpy(raw).to(DEV)
    if packed:
        iq3_pack.pack_(w, t)
    st = torch.cuda.current_stream().cuda_stream
    for m in (1, 4, 5, 8, 9, 12, 13, 16):
        x = synth.make_activation(m, k, 61 + m)
        q, d = q8_1.quantize_q8_1(x)[:2]
        want = product.product_q81(dec, q, d)
        xd = torch.from_numpy(x).to(DEV)
        q8 = torch.empty(m * k // 32 * 36, dtype=torch.uint8, device=DEV)
        assert lib.gsq_quantize_q8_1(xd.data_ptr(), 0, m, k, k, q8.data_ptr(), st) == 0
        y = torch.full((m + 1, rows + 5), float("nan"), device=DEV)
        assert lib.gsq_mul_mat_vec_q8(w.data_ptr(), w.shape[1], rows, t, int(packed), q8.data_ptr(), m, k, y.data_ptr(), 0, rows + 5, st) == 0
        assert bool(torch.isnan(y[:, rows:]).all()) and bool(torch.isnan(y[m]).all())
        # (fp32 sums in another order: 1e-7 measured)
        assert product.rel_err(y[:m, :rows].cpu().numpy(), want) <= 2e-6, m
