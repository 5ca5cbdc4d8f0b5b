"""The native host path (module _gsq_ops): its routing against the Python table that is API, and on the GPU the fused
layer of several runs against one product per run, direct calls against the custom ops."""

import threading
import time

import pytest
import torch
import torch.utils._python_dispatch

import gsq_b200  # noqa: F401
from gsq_b200 import _cabi, _gsq_ops, lcpp_ops, synth
from gsq_b200.quantization import iq3_pack, linear

TYPES = {**synth.TYPE_IDS, **synth.LOW_BIT_TYPE_IDS}


def test_native_routing_is_the_python_table():
    bad = []
    for t in TYPES.values():
        for packed in (False, True):
            pk = packed and t in iq3_pack.PACKABLE_TYPES
            for n in (1, 2, 3, 5, 6, 7, 8, 9, 16, 17, 32, 33, 48, 49, 300):
                for rows in (1024, 2048, 2049, 5120, 12288, 17408):
                    for k in (512, 5120, 17408):
                        want = linear._lcpp_op(n, t, rows, k, pk)
                        if pk and t == 14:
                            want = "gsq_mul_mat_vec_q6k_packed" if want == "lcpp_mul_mat_vec_q" else "gsq_mul_mat_q6k_packed"
                        if _gsq_ops.route(n, t, rows, k, pk) != want:
                            bad.append((n, t, rows, k, pk))
    assert not bad, bad[:5]


def test_native_errors_are_python_exceptions():
    x, w = torch.zeros(70, 512, dtype=torch.bfloat16), torch.zeros(16, 112, dtype=torch.uint8)
    with pytest.raises(NotImplementedError, match="no kernel for ggml type 29 at 70"):
        _gsq_ops.linear(x, w, 29, None, False)
    with pytest.raises(NotImplementedError, match="Unsupported GGUF quantization type"):
        _gsq_ops.linear(x, w, 8, None, False)
    with pytest.raises(RuntimeError, match="must be CUDA tensors"):
        _gsq_ops.linear_runs(x[:4], w, [0, 16, 112, 29], False)


def test_interpreter_runs_while_a_call_does():
    """A native call lets other Python threads run (an unquantised product on the host stands in for one that waits)."""
    x, w = torch.randn(512, 4096), torch.randn(4096, 4096)
    state = {"done": False}

    def work():
        state["t"] = -time.perf_counter()
        for _ in range(5):
            _gsq_ops.linear(x, w, 0, None, False)
        state["t"] += time.perf_counter()
        state["done"] = True

    old = torch.get_num_threads()
    torch.set_num_threads(1)
    try:
        thread, ticks = threading.Thread(target=work), 0
        thread.start()
        while not state["done"]:
            time.sleep(1e-3)
            ticks += 1
        thread.join()
    finally:
        torch.set_num_threads(old)
    # one tick a millisecond or so where the interpreter is free, about one per call (of 5) where it is not
    assert state["t"] < 0.1 or ticks > 20, (state["t"], ticks)


def _fused_layer(names, rows, k):
    layer, method = torch.nn.Module(), linear.GGUFLinearMethod(None)
    method.create_weights(layer, k, list(rows), k, sum(rows), torch.bfloat16)
    for i, (sid, name, r) in enumerate(zip("qkv", names, rows)):
        layer.weight.load_shard(torch.from_numpy(synth.make_weight(TYPES[name], r, k, 20 + i)).cuda(), sid)
        layer.weight_type.shard_weight_type[sid] = TYPES[name]
    method.process_weights_after_loading(layer)
    return layer, method


def test_a_layer_is_read_at_every_call(monkeypatch):
    """apply() follows a layer whose types or shard map change after its first call."""
    layer, method, calls = torch.nn.Module(), linear.GGUFLinearMethod(None), []
    method.create_weights(layer, 512, [32, 16, 16], 512, 64, torch.bfloat16)
    for sid, rows in zip("qkv", (32, 16, 16)):
        layer.weight.load_shard(torch.zeros(rows, 512 // 256 * 144, dtype=torch.uint8), sid)
        layer.weight_type.shard_weight_type[sid] = 12
    layer.weight_type.shard_weight_type["v"] = 23
    method._create_padded_weight_param(layer)
    monkeypatch.setattr(linear, "fused_mul_mat_gguf", lambda x, w, t, *a: calls.append(t) or x)
    monkeypatch.setattr(torch.ops._C_gguf, "gsq_linear_runs", lambda x, w, runs, packed: calls.append(runs) or x, raising=False)
    x, w, size = torch.zeros(1, 512, dtype=torch.bfloat16), layer.weight, 288
    assert w.shard_offset_map == {"q": (0, 32, size), "k": (32, 48, size), "v": (48, 64, size)}
    method.apply(layer, x)
    layer.weight_type.shard_weight_type["k"] = 23          # another type of one shard
    method.apply(layer, x)
    w.shard_offset_map["v"] = (48, 56, size)               # another shard map
    method.apply(layer, x)
    layer.weight_type.shard_weight_type.update(q=12, k=12, v=12)
    method.apply(layer, x)
    w.shard_id = []                                        # one product of the layer's own type
    layer.weight_type.weight_type = 21
    method.apply(layer, x)
    assert calls == [[0, 48, size, 12, 48, 16, size, 23], [0, 32, size, 12, 32, 32, size, 23], [0, 32, size, 12, 32, 24, size, 23], 12, 21]


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 4, 8, 9, 40, 70])
@pytest.mark.parametrize("names", [("IQ3_S", "IQ3_S", "Q6_K"), ("Q4_K", "IQ4_XS", "Q4_K"), ("IQ3_S", "IQ2_XS", "Q2_K")])
def test_runs_of_a_fused_layer(m, names):
    k, rows = 1024, (160, 48, 64)
    layer, method = _fused_layer(names, rows, k)
    x = torch.from_numpy(synth.make_activation(m, k, 30 + m)).to(torch.bfloat16).cuda()
    got = method.apply(layer, x)
    w = layer.weight
    packed = getattr(w, "iq3_packed", False)
    want = torch.cat([linear._fused_mul_mat_gguf(x, v, t, None, packed)
                      for v, t in linear._shard_runs(w, ["q", "k", "v"], [TYPES[n] for n in names])], dim=1)
    assert torch.equal(got, want)
    seen = []

    class Watch(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    with Watch():   # someone intercepts: through the custom op, same result
        assert torch.equal(method.apply(layer, x), want)
    assert "_C_gguf.gsq_linear_runs.default" in seen


@pytest.mark.gpu
@pytest.mark.parametrize("m", [1, 4, 40])
def test_output_into_of_a_fused_layer(m):
    """output_into holds for a layer whose shards are of several types: the caller's tensor, strided rows included, or an
    error if it does not fit."""
    k, rows = 1024, (160, 48, 64)
    layer, method = _fused_layer(("IQ3_S", "IQ3_S", "Q6_K"), rows, k)
    x = torch.from_numpy(synth.make_activation(m, k, 31)).to(torch.bfloat16).cuda()
    want = method.apply(layer, x)
    buf = torch.full((m, 300), -1.0, dtype=torch.bfloat16, device="cuda")
    into = buf[:, 8:8 + sum(rows)]
    with lcpp_ops.output_into(into):
        got = method.apply(layer, x)
    assert got.data_ptr() == into.data_ptr() and torch.equal(into, want)
    assert bool((buf[:, :8] == -1).all()) and bool((buf[:, 8 + sum(rows):] == -1).all())
    for bad in (torch.empty(m, 160, dtype=torch.bfloat16, device="cuda"), torch.empty(m, sum(rows), device="cuda")):
        with pytest.raises(RuntimeError, match="output_into"), lcpp_ops.output_into(bad):
            method.apply(layer, x)
    assert torch.equal(method.apply(layer, x), want)


@pytest.mark.gpu
@pytest.mark.parametrize("name,m", [("Q6_K", 128), ("IQ2_S", 64), ("IQ4_XS", 300)])
def test_short_of_memory(name, m):
    """Where the allocator has no room for expanded weights the product runs in the least scratch, with that form's result."""
    t, rows, k = TYPES[name], 4096, 17408
    w = torch.from_numpy(synth.make_weight(t, 64, k, 40)).cuda().repeat(rows // 64, 1)
    if t in iq3_pack.PACKABLE_TYPES:
        iq3_pack.pack_(w, t)
    packed, x = t in iq3_pack.PACKABLE_TYPES, torch.from_numpy(synth.make_activation(m, k, 41)).to(torch.bfloat16).cuda()
    lib = _cabi.lib
    most, least = lib.gsq_linear_workspace_bytes(rows, m, k, t, packed), lib.gsq_linear_scratch_bytes(rows, m, k, t, packed)
    assert most > (128 << 20) and least < (32 << 20)
    want, scratch = torch.empty(m, rows, dtype=torch.bfloat16, device="cuda"), torch.empty(least, dtype=torch.uint8, device="cuda")
    assert lib.gsq_linear(w.data_ptr(), w.shape[1], rows, t, packed, x.data_ptr(), _cabi.BF16, m, k, k, want.data_ptr(), _cabi.BF16, rows,
                          scratch.data_ptr(), least, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (100 << 20)) / total)
    try:
        got = _gsq_ops.linear(x, w, t, None, packed)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert torch.equal(got, want)
    torch.testing.assert_close(_gsq_ops.linear(x, w, t, None, packed).float(), want.float(), rtol=2e-2, atol=2e-2 * want.float().abs().mean().item())
