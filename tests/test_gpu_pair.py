"""Two products in one launch beyond contiguous bf16 X and fp32 Y: weight rows that are no multiple of 16, X of each type, padded and
unaligned, 16-bit Y with padded rows; and every pair of types through apply()."""

import numpy as np
import pytest
import torch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, synth
from gsq_b200.quantization import iq3_pack, linear
from oracle import blocks, product, q8_1

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = {"IQ3_S": 21, "IQ4_XS": 23, "Q4_K": 12, "Q6_K": 14}
PAIRS = [("Q4_K", "Q6_K"), ("IQ3_S", "Q6_K"), ("IQ4_XS", "Q6_K"), ("IQ3_S", "IQ4_XS")]
DTYPES = {"fp32": (0, torch.float32), "fp16": (1, torch.float16), "bf16": (2, torch.bfloat16)}
UNSUPPORTED = -3


def _packed(name):
    return int(name in ("IQ3_S", "Q6_K"))


@pytest.mark.parametrize("pair", PAIRS)
@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("k,pad,shift", [(256, 0, 0), (1280, 3, 1), (2560, 8, 0), (5120, 1, 3)])
def test_forms_of_x_and_y(pair, dtype, k, pad, shift):
    lib, st = _cabi.lib, torch.cuda.current_stream().cuda_stream
    code, tdt = DTYPES[dtype]
    rows = [r if _packed(n) else r - 11 for n, r in zip(pair, (1072, 272))]   # (repacked weights are whole 16-row records)
    raws = [synth.make_weight(TYPES[n], r, k, 120 + r) for n, r in zip(pair, rows)]
    ws = [torch.from_numpy(raw).to(DEV) for raw in raws]
    for n, w in zip(pair, ws):
        if _packed(n):
            iq3_pack.pack_(w, TYPES[n])
    total = sum(rows)
    for m in (4, 7, 8):
        x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 121 + m)).to(tdt))
        buf = torch.full((m * (k + pad) + shift,), float("nan"), dtype=tdt, device=DEV)   # shift: X itself is not 16-byte aligned
        buf[shift:].view(m, k + pad)[:, :k] = x.to(DEV)
        xp = buf.data_ptr() + shift * buf.element_size()
        q, d = q8_1.quantize_q8_1(x.float().numpy())[:2]
        want = np.concatenate([product.product_q81(blocks.decode(raw, TYPES[n]), q, d) for n, raw in zip(pair, raws)], axis=1)
        q8 = torch.empty(m * k // 32 * 36, dtype=torch.uint8, device=DEV)
        assert lib.gsq_quantize_q8_1(xp, code, m, k, k + pad, q8.data_ptr(), st) == 0
        for src, sdt, stride in ((q8.data_ptr(), -1, 0), (xp, code, k + pad)):
            got = {}
            for ycode, ydt in DTYPES.values():
                y = torch.full((m, total + 3), float("nan"), dtype=ydt, device=DEV)   # odd row stride
                a, b = (_cabi.Weight(w.data_ptr(), w.shape[1], r, TYPES[n], _packed(n), y.data_ptr() + c * y.element_size())
                        for n, w, r, c in zip(pair, ws, rows, (0, rows[0])))
                rc = lib.gsq_linear_vec_pair(a, b, src, sdt, m, k, stride, ycode, total + 3, st)
                if rc == UNSUPPORTED and sdt >= 0:
                    assert m * k > 10000   # (X is quantised inside while it is small)
                    break
                assert rc == 0, lib.gsq_strerror(rc)
                assert bool(torch.isnan(y[:, total:]).all())
                got[ydt] = y[:, :total]
            if got:
                # (fp32 sums in another order; the 16-bit results are those sums rounded once)
                assert product.rel_err(got[torch.float32].cpu().numpy(), want) <= 2e-6
                for ydt in (torch.float16, torch.bfloat16):
                    assert torch.equal(got[ydt], got[torch.float32].to(ydt))


def _layer(names, k, tdt):
    """A fused layer, q and k of the one type and v of the other; its rows' bytes."""
    shards = [("q", names[0], 1040), ("k", names[0], 256), ("v", names[1], 256)]
    layer, method = torch.nn.Module(), linear.GGUFLinearMethod(None)
    method.create_weights(layer, k, [r for _, _, r in shards], k, sum(r for _, _, r in shards), tdt)
    raws = []
    for i, (sid, name, rows) in enumerate(shards):
        raws.append((name, synth.make_weight(TYPES[name], rows, k, 130 + i)))
        layer.weight.load_shard(torch.from_numpy(raws[-1][1]).to(DEV), sid)
        layer.weight_type.shard_weight_type[sid] = TYPES[name]
    layer.weight_type.weight_type = TYPES[names[0]]
    method.process_weights_after_loading(layer)
    return layer, method, raws


@pytest.mark.parametrize("pair", PAIRS)
@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("order", [0, 1])
def test_through_apply(pair, dtype, order):
    """A fused layer of two types in either order (the pairs have one: the other is two launches)."""
    k, tdt = 2560, DTYPES[dtype][1]
    layer, method, raws = _layer(pair if order == 0 else pair[::-1], k, tdt)
    bound = {torch.float32: 1e-5, torch.float16: 1e-3, torch.bfloat16: 5e-3}[tdt]
    for m in (1, 2, 4, 7, 8):
        x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 131 + m)).to(tdt))
        q, d = q8_1.quantize_q8_1(x.float().numpy())[:2]
        want = np.concatenate([product.product_q81(blocks.decode(raw, TYPES[n]), q, d) for n, raw in raws], axis=1)
        wide = torch.empty((m, k + 24), dtype=tdt, device=DEV)
        wide[:, 16:16 + k] = x.to(DEV)
        for xd in (x.to(DEV), wide[:, 16:16 + k]):
            y = method.apply(layer, xd)
            assert y.dtype == tdt
            # 8 rows of some types go through the ops that read 128-value blocks (Q4_K's minimum from their half sums)
            assert product.rel_err(y.float().cpu().numpy(), want) <= max(bound, 1e-3 if m == 8 else 0), m


@pytest.mark.parametrize("pair", PAIRS)
@pytest.mark.parametrize("order", [0, 1])
def test_which_launches_apply_takes(pair, order, capfd):
    """One launch for both types in the pair's order, from the rows at which the small-batch kernel has both (Q4_K 2, IQ4_XS 4) to 7,
    whether X goes in itself or as blocks; replayed from a graph it gives the same."""
    k, lib = 2560, _cabi.lib
    layer, method, _ = _layer(pair if order == 0 else pair[::-1], k, torch.bfloat16)
    first = max({"Q4_K": 2, "IQ4_XS": 4}.get(n, 1) for n in pair)
    for m in range(1, 9):
        x = torch.from_numpy(synth.make_activation(m, k, 140 + m)).to(torch.bfloat16).to(DEV)
        method.apply(layer, x)
        capfd.readouterr()
        old = lib.gsq_debug_mmv_trace(1)
        y = method.apply(layer, x)
        lib.gsq_debug_mmv_trace(old)
        err = capfd.readouterr().err
        one = order == 0 and first <= m <= 7
        assert err.count("mmv pair") == int(one) and not (one and "mmv plan" in err), (m, err)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            got = method.apply(layer, x)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, y)
