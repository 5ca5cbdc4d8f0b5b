"""The two-step product (weights expanded to fp16 operand tiles, then the tcgen05 GEMM on pairs of CTAs): every weight
kind at the edges of its tiles (row tiles of 128 in pairs, token blocks of a multiple of 16, superblocks, parts of K),
against the float64 product of the dequantised weights and the q8_1 activations.

Q6_K, IQ3_S in GGUF order, Q2_K and IQ1_M keep exact integer slice sums and scale them in fp32, as their kernels of few rows
do: 2.5e-7 of a row's norm (rounding of 20 to 40 fp32 sums in a chain of chains is 1e-7 rms, that of the fp32 weights of
the oracle 3e-8, and a row of 16 results scatters by half). The other low-bit types carry 22 bits of d_x * q and exact
weights: 3e-6. (Their small-row kernels truncate integer divisions as the reference's do; the many-row form, like the
reference's, does not.)"""

import ctypes

import numpy as np
import pytest
import torch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, synth
from gsq_b200.quantization import iq3_pack
from oracle import blocks, blocks_f1, product, q8_1

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TYPES = {**synth.TYPE_IDS, **synth.LOW_BIT_TYPE_IDS}


def _run(t, packed, raw, x, rows, ldy=None, least=False):
    w = torch.from_numpy(raw).to(DEV)
    if packed:
        iq3_pack.pack_(w, t)
    lib, (m, k) = _cabi.lib, x.shape
    n = (lib.gsq_linear_scratch_bytes if least else lib.gsq_linear_workspace_bytes)(rows, m, k, t, int(packed))
    scratch = torch.full((n,), 0xFF, dtype=torch.uint8, device=DEV)     # nothing may rely on what it holds
    ldy = ldy or rows
    y = torch.full((m, ldy), float("nan"), dtype=torch.float32, device=DEV)
    rc = lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, int(packed), x.data_ptr(), 0, m, k, x.stride(0), y.data_ptr(), 0, ldy,
                        scratch.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, lib.gsq_strerror(rc)
    torch.cuda.synchronize()
    assert bool(torch.isnan(y[:, rows:]).all())
    flag = ctypes.c_int(-1)
    assert lib.gsq_device_error_flag(ctypes.byref(flag)) == 0 and flag.value == 0
    return y[:, :rows].cpu().numpy()


def _dense(raw, t):
    return product.product_full(raw, t, np.eye(_k(raw, t), dtype=np.float32)).T if t in synth.TYPE_IDS.values() else blocks_f1.product_full(
        raw, t, np.eye(_k(raw, t), dtype=np.float32)).T


def _k(raw, t):
    return raw.shape[1] // synth.BLOCK_BYTES[t] * 256


INTEGER_SUMS = ("Q6_K", "IQ3_S", "Q2_K", "IQ1_M")
CASES = [("Q6_K", True), ("Q6_K", False), ("IQ3_S", False)] + [(n, False) for n in synth.LOW_BIT_TYPE_IDS]


@pytest.mark.parametrize("name,packed", CASES)
@pytest.mark.parametrize("rows,k,m", [(16, 256, 130), (144, 512, 257), (400, 1024, 99), (272, 4608, 300)])
def test_full_precision_kinds(name, packed, rows, k, m):
    t = TYPES[name]
    raw = synth.make_weight(t, rows, k, 60 + rows)
    xa = synth.make_activation(m, k, 61 + m)
    xa[3, :64] = 0.0
    xa[7, :] = 0.0
    xa[5, 7] = 300.0
    x = synth.nudge_ties_torch(torch.from_numpy(xa).to(torch.bfloat16)).float()
    q, d, _ = q8_1.quantize_q8_1(x.numpy())
    xq = (q.reshape(m, k // 32, 32).astype(np.float64) * d.astype(np.float64).reshape(m, k // 32, 1)).reshape(m, k)
    want = xq @ _dense(raw, t).astype(np.float64).T
    got = _run(t, packed, raw, x.to(DEV), rows, rows + 5)
    assert np.isfinite(got).all() and not got[7].any()
    assert product.rel_err(got, want) <= (2.5e-7 if name in INTEGER_SUMS else 3e-6)


@pytest.mark.parametrize("name,packed", [c for c in CASES if c[0] in INTEGER_SUMS])
@pytest.mark.parametrize("m", [130, 131, 145, 160, 190, 256, 300])
def test_integer_sums_over_token_blocks(name, packed, m):
    """Every width of a warp's share of the tokens, K of one to four parts; the error is no larger than that of the kernels
    of few rows (their launches repeated: the INTEGER setting) beyond the scatter of 48 results a row."""
    t, rows, k = TYPES[name], 48, (256, 3072, 9216)[m % 3]
    raw = synth.make_weight(t, rows, k, 64 + m)
    x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 65 + m)).to(torch.bfloat16)).float()
    q, d, _ = q8_1.quantize_q8_1(x.numpy())
    xq = (q.reshape(m, k // 32, 32).astype(np.float64) * d.astype(np.float64).reshape(m, k // 32, 1)).reshape(m, k)
    want = xq @ _dense(raw, t).astype(np.float64).T

    def error():
        got = _run(t, packed, raw, x.to(DEV), rows)
        return np.linalg.norm(got - want) / np.linalg.norm(want)

    here, old = error(), _cabi.lib.gsq_prefill_precision(2)
    try:
        few = error()
    finally:
        _cabi.lib.gsq_prefill_precision(old)
    assert here <= 1.1 * few and few < 2e-7, (here, few)


def test_largest_integer_sums():
    """Q6_K at the ends of its fields: every slice sum is 128 * 32 * 127 * 32, just below 2^24."""
    rows, k, m = 32, 512, 97
    raw = synth.make_weight(14, rows, k, 66)
    blk = raw.reshape(rows, k // 256, 210)
    blk[:, :, :192] = 0          # q = -32
    blk[:, :, 192:208] = 0x80    # sub-scale -128
    x = torch.full((m, k), 127.0)
    x[1::2] = -127.0
    got = _run(14, True, raw, x.to(DEV), rows)
    d = np.ascontiguousarray(blk[:, :, 208:210]).view(np.float16)[..., 0].astype(np.float64).sum(1) * (8 * 128 * 32 * 127 * 32)
    want = np.where(np.arange(m)[:, None] % 2 == 0, d, -d)
    assert product.rel_err(got, want) <= 2e-7


@pytest.mark.parametrize("name,packed", CASES)
def test_numbers_that_are_not_finite(name, packed):
    """An infinite weight scale, a NaN and an infinity among the activations end where the kernels of few rows put them: a
    row that is not finite (infinite or NaN depends on where the scale is multiplied in), nothing (a NaN quantises to 0),
    a token that is not finite."""
    t, rows, k, m = TYPES[name], 32, 2048, 130
    raw = synth.make_weight(t, rows, k, 67)
    blk = raw.reshape(rows, k // 256, -1)
    at = {14: 208, 10: 80, 29: None}.get(t, 0)
    if at is not None:
        blk[3, 1, at:at + 2] = np.array([0x00, 0x7C], dtype=np.uint8)
    x = torch.from_numpy(synth.make_activation(m, k, 68)).float()
    x[2, 5] = float("nan")
    x[4, 300] = float("inf")
    got = _run(t, packed, raw, x.to(DEV), rows)
    old = _cabi.lib.gsq_prefill_precision(2)
    try:
        want = _run(t, packed, raw, x.to(DEV), rows)
    finally:
        _cabi.lib.gsq_prefill_precision(old)
    ok = np.isfinite(got)
    assert np.array_equal(ok, np.isfinite(want)) and not ok[4].any() and ok[2].sum() >= rows - 1
    assert at is None or not ok[:, 3].any()
    assert np.linalg.norm(got[ok] - want[ok]) <= 2e-4 * np.linalg.norm(want[ok])   # (truncating divisions: 5e-5)


def test_weights_expanded_in_several_chunks():
    """A weight above the bound on expanded weights goes a range of rows at a time through one buffer: results on both sides
    of each seam, and the whole against the same rows called by themselves."""
    t, rows, k, m = 14, 7680 + 272, 17408, 100
    assert rows * k * 4 > 512 << 20
    g = torch.Generator(DEV).manual_seed(93)
    w = torch.randint(0, 256, (rows, k // 256, 210), dtype=torch.uint8, device=DEV, generator=g)
    w[..., 208:210] = (torch.randn(rows, k // 256, device=DEV, generator=g).abs() * 1e-2).to(torch.float16).unsqueeze(-1).view(torch.uint8)
    w = w.view(rows, -1)
    sample = [0, 1, 6911, 6912, 7167, 7168, 7169, 7424, 7679, 7680, 7681, rows - 1]
    raw = w[sample].cpu().numpy()
    iq3_pack.pack_(w, t)
    x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 94)).to(torch.bfloat16)).float()
    lib, xd = _cabi.lib, x.to(DEV)

    def run(w):
        n = w.shape[0]
        size = lib.gsq_linear_workspace_bytes(n, m, k, t, 1)
        scratch = torch.full((size,), 0xFF, dtype=torch.uint8, device=DEV)
        y = torch.full((m, n), float("nan"), device=DEV)
        assert lib.gsq_linear(w.data_ptr(), w.shape[1], n, t, 1, xd.data_ptr(), 0, m, k, k, y.data_ptr(), 0, n, scratch.data_ptr(), size,
                              torch.cuda.current_stream().cuda_stream) == 0
        return y

    y = run(w)
    q, d, _ = q8_1.quantize_q8_1(x.numpy())
    assert product.rel_err(y[:, sample].cpu().numpy(), product.product_q81(blocks.decode(raw, t), q, d)) <= 2.5e-7
    for a in range(0, rows, 2048):
        part = run(w[a:a + 2048])
        assert bool(((part - y[:, a:a + 2048]).norm(dim=1) <= 2.5e-7 * part.norm(dim=1)).all())


@pytest.mark.parametrize("m", [256, 257, 272, 511, 529])
@pytest.mark.parametrize("name", ["IQ3_S", "IQ4_XS", "Q4_K"])
def test_rounded_kinds_over_token_blocks(name, m):
    """Ragged token counts and a K that is cut into parts: the model of the rounded form's own arithmetic."""
    from oracle import prefill_forms

    t, rows, k = TYPES[name], 400, 4096
    raw = synth.make_weight(t, rows, k, 70)
    x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 71 + m)).to(torch.bfloat16)).float()
    got = _run(t, name == "IQ3_S", raw, x.to(DEV), rows)
    assert product.rel_err(got, prefill_forms.product(raw, t, x.numpy())) <= 3e-6


def _integer_sums(raw, t, packed, x):
    """The arithmetic of the kernels with integer slice sums, the scaling in float64: 128-value blocks for repacked IQ3_S,
    IQ4_XS and Q4_K (there d, sum x, d * sc and dmin * m in half, as the int8 GEMM keeps them), block_q8_1 for the others."""
    dec = blocks.decode(raw, t)
    if t == 14 or (t == 21 and not packed):
        q, d, _ = q8_1.quantize_q8_1(x)
        return product.product_q81(dec, q, d)
    q, d, s = q8_1.quantize_mmq(x, q8_1.LAYOUT_DS4 if t == 12 else q8_1.LAYOUT_D4)
    if t == 12:
        f16, f64 = np.float16, np.float64
        scale, least = [(np.repeat(a, 8, axis=1).astype(f16) * i.astype(f16)).astype(f64) for a, i in ((dec.d, dec.isc), (dec.dmin, dec.imin))]
        y = np.einsum("mns,ns,ms->mn", product.block_sums(dec, q).astype(f64), scale, d.astype(f16).astype(f64), optimize=True)
        return y - s.astype(f16).astype(f64) @ least.T
    return product.product_q81(dec, q, d)


@pytest.mark.parametrize("name,packed,m", [("IQ3_S", True, 256), ("IQ4_XS", False, 300), ("Q4_K", False, 520), ("Q6_K", True, 99),
                                           ("Q6_K", False, 26)])
def test_least_scratch(name, packed, m):
    """A caller whose scratch has no room for expanded weights gets the kernels that need none."""
    t, rows, k = TYPES[name], 272, 1024
    raw = synth.make_weight(t, rows, k, 72)
    x = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(m, k, 73 + m)).to(torch.bfloat16)).float()
    lib = _cabi.lib
    assert lib.gsq_linear_scratch_bytes(rows, m, k, t, int(packed)) < lib.gsq_linear_workspace_bytes(rows, m, k, t, int(packed))
    got = _run(t, packed, raw, x.to(DEV), rows, least=True)
    assert product.rel_err(got, _integer_sums(raw, t, packed, x.numpy())) <= 2e-6


def test_long_prompt_with_k_in_parts():
    """More tokens than a grid's y takes, on a weight small enough that K is cut into parts whose sums a second kernel adds."""
    from oracle import prefill_forms

    name, rows, k, m = "IQ4_XS", 16, 5632, 65537
    t, lib = TYPES[name], _cabi.lib
    # (64 rows of this K are not cut; beside the parts their scratch is the same, one pair of row tiles)
    assert lib.gsq_linear_workspace_bytes(rows, m, k, t, 0) - lib.gsq_linear_workspace_bytes(64, m, k, t, 0) >= 2 * m * rows * 4
    raw = synth.make_weight(t, rows, k, 90)
    x = torch.randn(m, k, device=DEV, generator=torch.Generator(DEV).manual_seed(91), dtype=torch.bfloat16)
    at = [0, 1, 4095, 65534, 65535, 65536]
    few = synth.nudge_ties_torch(torch.from_numpy(synth.make_activation(len(at), k, 92)).to(torch.bfloat16))
    x[at] = few.to(DEV)
    w = torch.from_numpy(raw).to(DEV)
    y = torch.ops._C_gguf.lcpp_mul_mat_q(w, x, t, rows)
    got = y[at].float().cpu().numpy()
    assert bool(torch.isfinite(y).all())
    # 3e-6 for the sums, and the rounding of the result to bf16 (8 significant bits: at most 2^-8 of a value)
    assert product.rel_err(got, prefill_forms.product(raw, t, few.float().numpy())) <= 2.0 ** -8 + 3e-6


@pytest.mark.parametrize("m", [1, 40, 100, 300])
@pytest.mark.parametrize("name", ["Q4_K", "IQ4_XS"])
def test_packed_flag_on_a_type_of_one_layout(name, m):
    rows, k, t, lib = 24, 1024, TYPES[name], _cabi.lib
    w = torch.from_numpy(synth.make_weight(t, rows, k, 95)).to(DEV)
    x = torch.from_numpy(synth.make_activation(m, k, 96)).to(DEV)
    y = []
    for packed in (0, 1):
        n = lib.gsq_linear_workspace_bytes(rows, m, k, t, packed)
        scratch, out = torch.empty(n, dtype=torch.uint8, device=DEV), torch.empty(m, rows, device=DEV)
        assert lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, packed, x.data_ptr(), 0, m, k, k, out.data_ptr(), 0, rows, scratch.data_ptr(), n,
                              torch.cuda.current_stream().cuda_stream) == 0
        y.append(out)
    assert torch.equal(*y)


@pytest.mark.parametrize("name,rows,k,m", [("Q6_K", 848, 5120, 49), ("Q6_K", 2048, 5120, 96), ("Q6_K", 2064, 2560, 81), ("Q6_K", 8192, 1024, 96),
                                           ("IQ4_XS", 23, 512, 33), ("IQ4_XS", 1000, 1024, 48), ("IQ4_XS", 2049, 8448, 41), ("IQ4_XS", 1023, 17408, 48),
                                           ("Q4_K", 23, 256, 33), ("Q4_K", 777, 2048, 48), ("Q4_K", 5121, 5120, 41), ("Q4_K", 1000, 17408, 34)])
def test_row_counts_that_two_kernels_serve(name, rows, k, m):
    """33..48 rows of Q4_K and IQ4_XS, 49..96 of repacked Q6_K: the kernel that the rules choose against the other one that
    serves the same call. Both round K / 32 fp32 sums of exact integer products (Q4_K: twice as many, of terms that partly
    cancel): each is within sqrt(K / 32) of an fp32 rounding, 2^-24, and their difference within four times that."""
    t, packed, lib = TYPES[name], name == "Q6_K", _cabi.lib
    raw = synth.make_weight(t, rows, k, 69 + rows)
    x = torch.from_numpy(synth.make_activation(m, k, 70 + m)).float().to(DEV)
    x[m - 1, :64] = 0.0
    x[3, :] = 0.0
    here = _run(t, packed, raw, x, rows, rows + 3)
    if packed:
        old = lib.gsq_prefill_precision(2)
        other = _run(t, packed, raw, x, rows)
        lib.gsq_prefill_precision(old)
    else:
        old = lib.gsq_debug_gemm_variant(10)
        other = _run(t, packed, raw, x, rows)
        lib.gsq_debug_gemm_variant(old)
    assert not here[3].any() and np.isfinite(here).all()
    assert product.rel_err(here, other) <= 4 * np.sqrt(k / 32) * 2.0 ** -24
    if packed:
        assert np.array_equal(_run(t, packed, raw, x, rows, least=True), other)     # no room for expanded weights: launches
