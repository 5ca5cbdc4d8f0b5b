"""Small products that quantise X inside the product kernel: the quantiser kernels' values (so the two-call result up to the
order of the fp32 sums), ragged rows of Y and column counts, strided and unaligned X, each data type."""

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
DTYPES = {"fp32": (0, torch.float32), "fp16": (1, torch.float16), "bf16": (2, torch.bfloat16)}
UNSUPPORTED = -3


@pytest.mark.parametrize("name", list(TYPES))
@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("rows,k,ms", [(16, 256, (1, 5, 8, 16)), (1040, 2304, (1, 2, 7, 8, 9, 15)), (2064, 5120, (1, 3, 4))])
@pytest.mark.parametrize("pad", [0, 3])
def test_quantised_in_the_product(name, dtype, rows, k, ms, pad):
    t = TYPES[name]
    lib, code, tdt = _cabi.lib, DTYPES[dtype][0], DTYPES[dtype][1]
    raw = synth.make_weight(t, rows, k, 90 + rows)
    dec = blocks.decode(raw, t)
    w = torch.from_numpy(raw).to(DEV)
    packed = name in ("IQ3_S", "Q6_K")
    if packed:
        iq3_pack.pack_(w, t)
    st = torch.cuda.current_stream().cuda_stream
    for m in ms:
        xa = synth.make_activation(m, k, 91 + m)
        xa[0, :64] = 0.0
        xa[m - 1, 40] = 300.0
        x = synth.nudge_ties_torch(torch.from_numpy(xa).to(tdt))
        buf = torch.empty((m, k + pad), dtype=tdt, device=DEV)   # pad: rows that are not 16-byte aligned
        buf[:, :k] = x.to(DEV)
        xn = x.float().numpy()
        if m <= 8:
            y = torch.full((m, rows + 3), float("nan"), dtype=torch.float32, device=DEV)
            rc = lib.gsq_linear_vec(w.data_ptr(), w.shape[1], rows, t, int(packed), buf.data_ptr(), code, m, k, k + pad, y.data_ptr(), 0,
                                    rows + 3, st)
            if rc == UNSUPPORTED:   # the dp4a kernel's products
                assert name in ("IQ4_XS", "Q4_K") and rows > 2000 and m < 4 or m * k > 10000
            else:
                assert rc == 0, lib.gsq_strerror(rc)
                q, d = q8_1.quantize_q8_1(xn)[:2]
                want = product.product_q81(dec, q, d)
                assert bool(torch.isnan(y[:, rows:]).all())
                assert product.rel_err(y[:, :rows].cpu().numpy(), want) <= 2e-6
        layout = q8_1.LAYOUT_DS4 if name == "Q4_K" else q8_1.LAYOUT_D4
        q, d, s = q8_1.quantize_mmq(xn, layout)
        n = lib.gsq_linear_workspace_bytes(rows, m, k, t, int(packed))
        scratch = torch.full((n,), 0xFF, dtype=torch.uint8, device=DEV)
        y = torch.full((m, rows + 3), float("nan"), dtype=torch.float32, device=DEV)
        rc = lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, int(packed), buf.data_ptr(), code, m, k, k + pad, y.data_ptr(), 0, rows + 3,
                            scratch.data_ptr(), n, st)
        assert rc == 0, lib.gsq_strerror(rc)
        if name == "Q4_K":
            want = product.product_xsum(dec, q, d.astype(np.float16), s.astype(np.float16))
        else:
            want = product.product_q81(dec, q, d)
        assert bool(torch.isnan(y[:, rows:]).all())
        assert product.rel_err(y[:, :rows].cpu().numpy(), want) <= 2e-6


@pytest.mark.parametrize("name,ms", [("Q4_K", (1,)), ("IQ4_XS", (1, 2, 3))])
@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("rows,k,pad", [(12301, 256, 0), (3077, 1280, 1), (2050, 5120, 8), (516, 8192, 0), (516, 8448, 3)])
def test_dp4a_product_quantises_as_the_kernel_in_front(name, ms, dtype, rows, k, pad):
    """The dp4a kernel with X quantised inside: bit for bit what the quantiser kernel and the product on its blocks give."""
    t = TYPES[name]
    lib, code, tdt = _cabi.lib, DTYPES[dtype][0], DTYPES[dtype][1]
    w = torch.from_numpy(synth.make_weight(t, rows, k, 95 + rows)).to(DEV)
    st = torch.cuda.current_stream().cuda_stream
    for m in ms:
        buf = torch.empty((m, k + pad), dtype=tdt, device=DEV)
        buf[:, :k] = torch.from_numpy(synth.make_activation(m, k, 96 + m)).to(tdt).to(DEV)
        buf[0, :64] = 0.0
        out = [torch.full((m, rows + 3), float("nan"), dtype=torch.float32, device=DEV) for _ in range(2)]
        args = (w.data_ptr(), w.shape[1], rows, t, 0)
        rc = lib.gsq_linear_vec(*args, buf.data_ptr(), code, m, k, k + pad, out[0].data_ptr(), 0, rows + 3, st)
        if m * k > 8192:   # (the two calls are faster)
            assert rc == UNSUPPORTED
            continue
        assert rc == 0, lib.gsq_strerror(rc)
        q8 = torch.empty(m * k // 32 * 36, dtype=torch.uint8, device=DEV)
        assert lib.gsq_quantize_q8_1(buf.data_ptr(), code, m, k, k + pad, q8.data_ptr(), st) == 0
        assert lib.gsq_mul_mat_vec_q8(*args, q8.data_ptr(), m, k, out[1].data_ptr(), 0, rows + 3, st) == 0
        if rows * k > 3 << 20:   # (smaller ones: the tensor-core kernel, which adds in another order)
            assert torch.equal(out[0][:, :rows], out[1][:, :rows])
        assert product.rel_err(out[0][:, :rows].cpu().numpy(), out[1][:, :rows].cpu().numpy().astype(np.float64)) <= 1e-6
        assert bool(torch.isnan(out[0][:, rows:]).all())


@pytest.mark.parametrize("name,m,rows,inside", [("Q4_K", 1, 2064, False), ("Q4_K", 1, 13312, True), ("IQ4_XS", 1, 2064, False), ("IQ4_XS", 1, 13312, False)])
def test_dp4a_product_in_a_capture(name, m, rows, inside):
    """A capture takes the quantiser and the product as two kernels (but for the largest Q4_K); its replay gives what calls one by
    one give, bit for bit."""
    from gsq_b200 import _gsq_ops

    t, k = TYPES[name], 5120
    w = torch.from_numpy(synth.make_weight(t, rows, k, 77)).to(DEV)
    x = torch.from_numpy(synth.make_activation(m, k, 78)).to(torch.bfloat16).to(DEV)
    y = torch.empty((m, rows), dtype=torch.bfloat16, device=DEV)

    def vec():
        return _cabi.lib.gsq_linear_vec(w.data_ptr(), w.shape[1], rows, t, 0, x.data_ptr(), 2, m, k, k, y.data_ptr(), 2, rows,
                                        torch.cuda.current_stream().cuda_stream)

    assert vec() == 0
    eager = _gsq_ops.linear(x, w, t, None, False)
    assert torch.equal(eager, y)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        rc = vec()
        got = _gsq_ops.linear(x, w, t, None, False)
    assert rc == (0 if inside else UNSUPPORTED)
    g.replay()
    assert torch.equal(got, eager)


@pytest.mark.parametrize("pair", [("Q4_K", "Q6_K"), ("IQ3_S", "Q6_K"), ("IQ4_XS", "Q6_K"), ("IQ3_S", "IQ4_XS")])
@pytest.mark.parametrize("rows,k", [((16, 16), 256), ((48, 2064), 768), ((6144, 1024), 5120), ((1024, 34816), 2560), ((512, 256), 17408)])
def test_two_products_in_one_launch(pair, rows, k):
    """A fused layer of two types in one launch: what a call per type gives, up to the order of the fp32 sums; from blocks and, where
    both products take X, from X."""
    lib, st = _cabi.lib, torch.cuda.current_stream().cuda_stream
    raws = [synth.make_weight(TYPES[n], r, k, 97 + r) for n, r in zip(pair, rows)]
    ws = [torch.from_numpy(raw).to(DEV) for raw in raws]
    for n, w in zip(pair, ws):
        if n in ("IQ3_S", "Q6_K"):
            iq3_pack.pack_(w, TYPES[n])
    total = sum(rows)
    for m in (1, 2, 4, 7, 8):
        x = torch.from_numpy(synth.make_activation(m, k, 98 + m)).to(torch.bfloat16).to(DEV)
        q8 = torch.empty(m * k // 32 * 36, dtype=torch.uint8, device=DEV)
        assert lib.gsq_quantize_q8_1(x.data_ptr(), 2, m, k, k, q8.data_ptr(), st) == 0
        want = torch.full((m, total + 1), float("nan"), device=DEV)
        y = [torch.full_like(want, float("nan")) for _ in range(2)]

        def weights(out):
            return [_cabi.Weight(w.data_ptr(), w.shape[1], r, TYPES[n], int(n in ("IQ3_S", "Q6_K")), out.data_ptr() + 4 * c)
                    for n, w, r, c in zip(pair, ws, rows, (0, rows[0]))]

        for g in weights(want):
            assert lib.gsq_mul_mat_vec_q8(g.w, g.row_bytes, g.rows, g.ggml_type, g.packed, q8.data_ptr(), m, k, g.y, 0, total + 1, st) == 0
        a, b = weights(y[0])
        served = lib.gsq_linear_vec_pair_serves(a, b, m)
        rc = lib.gsq_linear_vec_pair(a, b, q8.data_ptr(), -1, m, k, 0, 0, total + 1, st)
        assert rc == (0 if served else UNSUPPORTED)
        a, b = weights(y[1])
        rx = lib.gsq_linear_vec_pair(a, b, x.data_ptr(), 2, m, k, k, 0, total + 1, st)
        assert rx in (0, UNSUPPORTED) and (rx == UNSUPPORTED or served)
        for code, got in ((rc, y[0]), (rx, y[1])):
            if code == 0:
                assert bool(torch.isnan(got[:, total:]).all())
                for c, r in ((0, rows[0]), (rows[0], rows[1])):
                    assert product.rel_err(got[:, c:c + r].cpu().numpy(), want[:, c:c + r].cpu().numpy().astype(np.float64)) <= 1e-6
            else:
                assert bool(torch.isnan(got).all())
