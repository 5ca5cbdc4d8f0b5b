"""What a user of the quantised-linear path has it do, as measurable cases.

A case is a dict of plain values with a `kind`:

  linear   one layer through GGUFLinearMethod.apply(): a single weight, or (several entries in `types` / `rows`) a fused
           layer whose shards are of one type or of several
  mlp      the MLP half of a decoder layer at decode row counts: RMSNorm + quantise, gate/up product, SwiGLU + quantise,
           down product (gsq_b200.fused and torch.ops.vllm._fused_mul_mat_gguf with the shared quantised activations)
  stack    the four linears of a decoder layer (qkv, o, gate/up, down), replayed from a CUDA graph, as a serving engine
           runs its decode step

`m` is the number of activation rows: tokens of a prompt, or sequences (times verify tokens) of a decode step. Weights are
seeded random blocks whose fields have the distributions of gsq_b200.synth, made on the GPU; activations are normal with
0.1 % of the entries twenty times larger, as the prefill configuration has them.
"""

import math
import os
import sys

import torch

_PKG = os.path.join(os.getcwd(), "vllm-gsqrco-exl3_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from gsq_b200 import fused  # noqa: E402
from gsq_b200.quantization import linear  # noqa: E402

TYPES = {"Q4_K": 12, "Q6_K": 14, "IQ3_S": 21, "IQ4_XS": 23,
         "Q2_K": 10, "IQ2_XXS": 16, "IQ2_XS": 17, "IQ3_XXS": 18, "IQ2_S": 22, "IQ1_M": 29}
BLOCK_BYTES = {"Q4_K": 144, "Q6_K": 210, "IQ3_S": 110, "IQ4_XS": 136,
               "Q2_K": 84, "IQ2_XXS": 66, "IQ2_XS": 74, "IQ3_XXS": 98, "IQ2_S": 82, "IQ1_M": 56}
MAIN = ("Q4_K", "Q6_K", "IQ3_S", "IQ4_XS")
LOW_BIT = ("Q2_K", "IQ2_XXS", "IQ2_XS", "IQ3_XXS", "IQ2_S", "IQ1_M")
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
DTYPE_BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}

# the decoder layer of the configurations: hidden 5120, 40 / 8 heads of 128, intermediate 17408, vocabulary 151936
HIDDEN, INTER, VOCAB = 5120, 17408, 151936
QKV = (5120, 1024, 1024)


def _linear(name, types, rows, k, m, dtype):
    return {"name": name, "kind": "linear", "types": types, "rows": rows, "k": k, "m": m, "dtype": dtype}


def listed():
    return [
        # one token of one sequence through the smallest linear of the row sweep: latency and launches
        _linear("decode1_q4k_5120", "Q4_K", "5120", 5120, 1, "fp16"),
        # the single-layer configuration: IQ3_S 17408 x 5120, one fp32 token
        _linear("decode1_iq3s_fp32", "IQ3_S", "17408", 5120, 1, "fp32"),
        # one sequence with 3 verify tokens: a fused qkv whose v shard is kept at a higher precision than q and k
        _linear("decode4_qkv_mixed", "IQ3_S,IQ3_S,Q6_K", "5120,1024,1024", 5120, 4, "bf16"),
        # two sequences with 3 verify tokens: the MLP half of a layer with the norms fused into the quantiser
        {"name": "decode8_mlp", "kind": "mlp", "up": "IQ3_S", "down": "IQ4_XS", "hidden": HIDDEN, "inter": INTER, "m": 8, "dtype": "bf16"},
        # eight sequences with 3 verify tokens: the linears of a decoder layer inside the engine's graph
        {"name": "decode32_stack", "kind": "stack", "attn": "IQ3_S", "down": "IQ4_XS", "hidden": HIDDEN, "inter": INTER, "m": 32, "dtype": "bf16"},
        # the logits of 16 rows: Q6_K head over the whole vocabulary
        _linear("head16_q6k", "Q6_K", "151936", 5120, 16, "bf16"),
        # a large decode batch / a short prompt, ragged
        _linear("batch100_iq4xs", "IQ4_XS", "5120", 17408, 100, "bf16"),
        # an ordinary prompt of an odd length
        _linear("prefill777_q4k", "Q4_K", "17408", 5120, 777, "fp16"),
        # prompts of the prefill configuration
        _linear("prefill2048_iq3s", "IQ3_S", "17408", 5120, 2048, "bf16"),
        _linear("prefill8192_iq4xs", "IQ4_XS", "5120", 17408, 8192, "bf16"),
        # files that keep down_proj or attn_v at 6 bits: the same prompts meet Q6_K
        _linear("prefill512_q6k", "Q6_K", "5120", 17408, 512, "bf16"),
        # and the low-bit types a mixed file has beside the four main ones
        _linear("prefill256_iq2s", "IQ2_S", "17408", 5120, 256, "bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dtype(rng):
    return rng.choice(["bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])


def _rows(rng, lo, hi):
    """Weight rows: multiples of 16 (a tensor-parallel shard is one), every fourth time one of the model's own."""
    if rng.random() < 0.25:
        return rng.choice([r for r in (1024, 2048, 5120, 7168, 17408, 34816) if lo <= r <= hi])
    return max(16, _log_int(rng, lo, hi) // 16 * 16)


def _cols(rng, lo, hi):
    """Columns: multiples of 512, which the ops demand."""
    if rng.random() < 0.25:
        return rng.choice([c for c in (2048, 5120, 17408) if lo <= c <= hi])
    return max(512, _log_int(rng, lo, hi) // 512 * 512)


def draw(rng):
    """Another case of the same ranges: decode of 1 to 48 rows, batches of 49 to 255, prompts of 256 to 8192 tokens on the
    four main types; the low-bit types from 1 to 512 rows (IQ1_M to 32, where its ops end)."""
    kind = rng.choice(["decode", "decode", "qkv", "mlp", "stack", "head", "batch", "batch", "prefill", "prefill", "prefill",
                       "low_bit", "low_bit"])
    if kind in ("decode", "batch", "prefill"):
        t = rng.choice(MAIN)
        lo, hi = {"decode": (1, 48), "batch": (49, 255), "prefill": (256, 8192)}[kind]
        m = _log_int(rng, lo, hi)
        n, k = _rows(rng, 512, 34816), _cols(rng, 1024, 17408)
        most = 8192 * 5120 * 17408 // (12 if t == "Q6_K" else 1)
        while m * n * k > most:
            m = max(lo, m // 2)
            if m == lo:
                n = max(16, n // 32 * 16)
        c = _linear("", t, str(n), k, m, _dtype(rng))
    elif kind == "low_bit":
        t = rng.choice(LOW_BIT)
        m = _log_int(rng, 1, 32 if t == "IQ1_M" else 512)
        n, k = _rows(rng, 512, 17408), _cols(rng, 1024, 17408)
        while m * n * k > 256 * 5120 * 17408:
            n = max(16, n // 32 * 16)
        c = _linear("", t, str(n), k, m, _dtype(rng))
    elif kind == "qkv":
        a, b = rng.choice([("IQ3_S", "Q6_K"), ("Q4_K", "Q6_K"), ("IQ4_XS", "Q6_K"), ("IQ3_S", "IQ4_XS"), ("IQ3_S", "IQ3_S"),
                           ("Q4_K", "Q4_K")])
        kv = rng.choice([256, 512, 1024, 2048])
        q = kv * rng.choice([2, 4, 5, 8])
        c = _linear("", "%s,%s,%s" % (a, a, b), "%d,%d,%d" % (q, kv, kv), _cols(rng, 1024, 8192), _log_int(rng, 1, 64), _dtype(rng))
    elif kind == "head":
        c = _linear("", "Q6_K", str(rng.choice([VOCAB, VOCAB // 2, VOCAB // 4, 32000, 128256])), _cols(rng, 1024, 5120), _log_int(rng, 1, 48),
                    rng.choice(["bf16", "fp16"]))
    else:
        hidden = _cols(rng, 1024, 6144)
        inter = max(1024, int(hidden * rng.uniform(2.5, 4.0)) // 512 * 512)
        down = rng.choice(["IQ4_XS", "Q4_K", "IQ3_S", "Q6_K"])
        up = rng.choice(["IQ3_S", "Q4_K"])
        if kind == "mlp":
            c = {"kind": "mlp", "up": up, "down": down, "hidden": hidden, "inter": inter, "m": rng.randint(1, 8), "dtype": rng.choice(["bf16", "fp16"])}
        else:
            c = {"kind": "stack", "attn": up, "down": down, "hidden": hidden, "inter": inter, "m": _log_int(rng, 1, 48), "dtype": rng.choice(["bf16", "fp16"])}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _half_bytes(shape, mult, g):
    return (torch.randn(shape, device="cuda", generator=g).abs_() * mult).to(torch.float16).unsqueeze(-1).view(torch.uint8)


def _weight(t, rows, k, g):
    """uint8 [rows, row_bytes] of valid blocks: uniform quants, indices, signs and sub-scales, normal super-block scales."""
    nb, bs = k // 256, BLOCK_BYTES[t]
    w = torch.randint(0, 256, (rows, nb, bs), dtype=torch.uint8, device="cuda", generator=g)
    mult = {"IQ3_S": 2e-3, "IQ4_XS": 1e-2, "Q4_K": 1e-2, "Q6_K": 1e-2}.get(t, 5e-3)
    if t == "IQ1_M":  # the four nibbles of d are the top nibbles of the block's four scale words
        d = _half_bytes((rows, nb), mult, g).to(torch.int32)
        d = d[..., 0] | d[..., 1] << 8
        for j in range(4):
            w[..., 49 + 2 * j] = ((w[..., 49 + 2 * j].to(torch.int32) & 0x0F) | ((d >> 4 * j) & 0xF) << 4).to(torch.uint8)
        return w.view(rows, nb * bs)
    for at in {"Q4_K": (0, 2), "Q6_K": (208,), "Q2_K": (80, 82)}.get(t, (0,)):
        w[..., at:at + 2] = _half_bytes((rows, nb), mult, g)
    return w.view(rows, nb * bs)


def _activations(m, k, dtype, g):
    x = torch.randn(m, k, device="cuda", generator=g)
    x = torch.where(torch.rand(m, k, device="cuda", generator=g) < 1e-3, x * 20, x)
    return x.to(DTYPES[dtype])


def _layer(types, rows, k, dtype, g):
    """(method, layer) as a model loader leaves them: shards loaded, padded, repacked."""
    layer, method = torch.nn.Module(), linear.GGUFLinearMethod(None)
    method.create_weights(layer, k, list(rows), k, sum(rows), DTYPES[dtype])
    ids = [None] if len(rows) == 1 else ["q", "k", "v"] if len(rows) == 3 else list(range(len(rows)))
    for i, t, n in zip(ids, types, rows):
        layer.weight.load_shard(_weight(t, n, k, g), i)
        if i is not None:
            layer.weight_type.shard_weight_type[i] = TYPES[t]
    layer.weight_type.weight_type = TYPES[types[0]]
    method.process_weights_after_loading(layer)
    return method, layer


def _shards(case):
    return case["types"].split(","), [int(r) for r in case["rows"].split(",")]


def _linears(case):
    """(types, rows, k) of each linear of a stack or an mlp case."""
    h, i = case["hidden"], case["inter"]
    if case["kind"] == "mlp":
        return [([case["up"]] * 2, [i, i], h), ([case["down"]], [h], i)]
    a = case["attn"]
    kv = max(128, h // 5 // 16 * 16)
    return [([a] * 3, [h, kv, kv], h), ([a], [h], h), ([a] * 2, [i, i], h), ([case["down"]], [h], i)]


def prepare(case, seed):
    g = _gen(seed)
    m, dtype = case["m"], case["dtype"]
    if case["kind"] == "linear":
        types, rows = _shards(case)
        method, layer = _layer(types, rows, case["k"], dtype, g)
        return {"kind": "linear", "method": method, "layer": layer, "x": _activations(m, case["k"], dtype, g)}
    layers = [_layer(t, r, k, dtype, g) for t, r, k in _linears(case)]
    if case["kind"] == "mlp":
        gamma = (1 + 0.1 * torch.randn(case["hidden"], device="cuda", generator=g)).to(DTYPES[dtype])
        return {"kind": "mlp", "up": layers[0][1], "down": layers[1][1], "gamma": gamma, "x": _activations(m, case["hidden"], dtype, g)}
    xs = [_activations(m, k, dtype, g) for _, _, k in _linears(case)]
    step = lambda: [method.apply(layer, x) for (method, layer), x in zip(layers, xs)]  # noqa: E731
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = step()
    return {"kind": "stack", "graph": graph, "outs": outs, "keep": (layers, xs)}


def _product(layer, x, x_q8):
    """A one-run layer on activations that are quantised already."""
    w = layer.weight
    t = layer.weight_type
    wt = t.shard_weight_type.get(w.shard_id[0], t.weight_type) if w.shard_id else t.weight_type
    return linear.fused_mul_mat_gguf(x, w, wt, x_q8, getattr(w, "iq3_packed", False))


def run(state):
    if state["kind"] == "linear":
        return state["method"].apply(state["layer"], state["x"])
    if state["kind"] == "stack":
        state["graph"].replay()
        return state["outs"]
    q8, y = fused.rmsnorm_quantize_q8_1(state["x"], state["gamma"], 1e-6, want_y=True)
    gate_up = _product(state["up"], y, q8)
    q8, act = fused.silu_mul_quantize_q8_1(gate_up, want_y=True)
    return _product(state["down"], act, q8), gate_up


def _one(types, rows, k, m, size):
    weight = sum(n * (k // 256) * BLOCK_BYTES[t] for t, n in zip(types, rows))
    n = sum(rows)
    return weight + (m * k + m * n) * size, 2.0 * m * n * k


def work(case):
    """Weights, activations in and results out once each; two operations per weight and row. For an mlp the activations
    between its two products are written and read once (they are what its entry points return and take)."""
    size, m = DTYPE_BYTES[case["dtype"]], case["m"]
    parts = [_shards(case) + (case["k"],)] if case["kind"] == "linear" else _linears(case)
    got = [_one(t, r, k, m, size) for t, r, k in parts]
    return {"bytes": float(sum(b for b, _ in got)), "flops": float(sum(f for _, f in got))}


def tolerance(case):
    """16-bit results: the rounding of the type itself (half an ulp apart at most places). fp32 results: sums of exact
    integer products up to 48 rows; above, the prefill products form d_x * q in fp16 operands unless the caller asks for
    more, which the path states as 1e-3 of a row's norm. The low-bit types' integer divisions truncate in one form of their
    product and not in another."""
    if case["dtype"] == "bf16":
        return {"rel": 5e-3}
    if case["dtype"] == "fp16":
        return {"rel": 1e-3}
    few = case["m"] <= 48 and all(t in MAIN for t in _shards(case)[0])
    return {"rel": 2e-5 if few else 1e-3}
