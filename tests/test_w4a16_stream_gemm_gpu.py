"""The two-pass int4 GEMM (csrc/w4a16_stream_gemm.cu) against the oracle's weight: one and many stream tiles, ragged
token counts, small and large groups, a bias, and the dispatch of AWQLinearMethod.

Bound: the weight is the oracle's bit by bit, so an element is off by one rounding of the result (2^-8 bf16, 2^-11 f16)
and fp32 sums of K products in any order (K * 2^-24 of the sum of magnitudes)."""
import pytest
import torch

from oracle import int4 as OI

pytestmark = pytest.mark.gpu


def _packed(k, n, group, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda rows: torch.randint(-2 ** 31, 2 ** 31, (rows, n // 8), device="cuda", generator=g).to(torch.int32)
    scales = ((torch.rand(k // group, n, device="cuda", generator=g) + 0.5) * 0.01).to(dtype)
    return draw(k), draw(k // group), scales, g


def _check(out, x, w, bias):
    ref = x.double() @ w.double() + (0 if bias is None else bias.double())
    mags = x.double().abs() @ w.double().abs() + (0 if bias is None else bias.double().abs())
    ulp = 2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -11
    assert bool(((out.double() - ref).abs() <= ulp * ref.abs() + (x.shape[1] * 2.0 ** -24 + 2.0 ** -22) * mags + 2.0 ** -24).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,group", [(1, 16, 64, 64), (33, 48, 128, 8), (257, 272, 640, 32), (700, 1040, 1152, 128),
                                         (513, 256, 4096, 4096)])
def test_matches_oracle_weight(m, n, k, group, dtype):
    from sglang_security_b200.layers.quantization.w4a16_kernel import gemv_stream_repack, unpack_zeros, w4a16_gemm_stream

    q, z, s, g = _packed(k, n, group, dtype, m + n + k)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    zeros = unpack_zeros(z, dtype, awq_order=True, add_one=False)
    w = OI.awq_dequantize_oracle(q, s, z, group)
    for b in (None, bias):
        _check(w4a16_gemm_stream(x, gemv_stream_repack(q), zeros, s, group, b), x, w, b)


@pytest.mark.parametrize("m,two_pass", [(512, False), (513, True), (1500, True)])
def test_layer_dispatch(m, two_pass):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.linear import ColumnParallelLinear
    from sglang_security_b200.layers.quantization.awq import AWQConfig

    k, n, dtype = 2048, 1024, torch.float16               # 2^21 weights: the smallest that are expanded
    q, z, s, g = _packed(k, n, 128, dtype, m)
    layer = ColumnParallelLinear(k, n, bias=False, params_dtype=dtype, quant_config=AWQConfig(4, 128, True), tp_rank=0,
                                 tp_size=1).cuda()
    layer.qweight.data.copy_(q)
    layer.qzeros.data.copy_(z)
    layer.scales.data.copy_(s)
    layer.quant_method.process_weights_after_loading(layer)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    out, _ = layer(x)
    assert _lib.last_variant().endswith("expanded") == two_pass, _lib.last_variant()
    _check(out, x, OI.awq_dequantize_oracle(q, s, z, 128), None)
    wide = torch.randn(m, k + 4, device="cuda", generator=g).to(dtype)[:, :k]     # rows the copies cannot start on
    out, _ = layer(wide.contiguous())
    _check(out, wide, OI.awq_dequantize_oracle(q, s, z, 128), None)


def test_no_room_for_the_expanded_weight(monkeypatch):
    """The layer still runs, on the fused kernel, where the scratch tensor cannot be had."""
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization import w4a16_kernel as W

    k, n, m, dtype = 2048, 1024, 1500, torch.float16
    q, z, s, g = _packed(k, n, 128, dtype, 5)
    layer = torch.nn.Module()
    layer.qweight, layer.scales, layer.w4a16_group_size = q, s, 128
    layer.b200_zeros = W.unpack_zeros(z, dtype, awq_order=True, add_one=False)
    layer.b200_qweight_stream = W.gemv_stream_repack(q)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)

    def refuse(*a, **kw):
        raise torch.cuda.OutOfMemoryError("no room")

    monkeypatch.setattr(W, "w4a16_gemm_stream", refuse)
    out = W.w4a16_linear(x, layer, None)
    assert not _lib.last_variant().endswith("expanded")
    _check(out, x, OI.awq_dequantize_oracle(q, s, z, 128), None)


def _awq_layer(k, n, dtype, seed):
    from sglang_security_b200.layers.linear import ColumnParallelLinear
    from sglang_security_b200.layers.quantization.awq import AWQConfig

    q, z, s, g = _packed(k, n, 128, dtype, seed)
    layer = ColumnParallelLinear(k, n, bias=False, params_dtype=dtype, quant_config=AWQConfig(4, 128, True), tp_rank=0,
                                 tp_size=1).cuda()
    for p, v in ((layer.qweight, q), (layer.qzeros, z), (layer.scales, s)):
        p.data.copy_(v)
    layer.quant_method.process_weights_after_loading(layer)
    return layer, OI.awq_dequantize_oracle(q, s, z, 128), g


def test_scratch_is_taken_with_the_weights_and_given_back():
    """A call allocates its output and no more; all layers of the device hold the same memory, also a copied and an
    unpickled one; it grows with a larger weight and goes with the last layer."""
    import copy
    import gc
    import pickle

    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization.w4a16_kernel import ExpandScratch

    gc.collect()
    dtype, m = torch.float16, 1500
    a, wa, g = _awq_layer(2048, 1024, dtype, 1)
    scratch = a.b200_expand_scratch
    assert scratch.size() >= 2048 * 1024 * 2
    b, wb, _ = _awq_layer(2048, 4096, dtype, 2)
    assert b.b200_expand_scratch is scratch and scratch.size() >= 2048 * 4096 * 2
    assert copy.deepcopy(scratch) is scratch and pickle.loads(pickle.dumps(scratch)) is scratch
    x = torch.randn(m, 2048, device="cuda", generator=g).to(dtype)
    for layer, w, n in ((a, wa, 1024), (b, wb, 4096)):
        out, _ = layer(x)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        again, _ = layer(x)
        assert torch.cuda.max_memory_allocated() - before <= m * n * 2 + 4096
        assert _lib.last_variant().endswith("expanded")
        assert torch.equal(out, again)
        _check(out, x, w, None)
    small, _, _ = _awq_layer(512, 1024, dtype, 3)
    assert small.b200_expand_scratch is None                              # never expanded
    held = torch.cuda.memory_allocated()
    size = scratch.size()
    del a, b, layer, scratch
    gc.collect()
    assert torch.device("cuda", 0).index not in ExpandScratch._of_device and torch.cuda.memory_allocated() <= held - size


def test_no_room_when_the_weights_were_loaded(monkeypatch):
    """The fused kernel runs, and the allocator is not asked for the expanded weight again."""
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization import w4a16_kernel as W

    real = torch.empty
    asked = []

    def empty(*a, **kw):
        if kw.get("dtype") == torch.uint8:
            asked.append(a)
            raise torch.cuda.OutOfMemoryError("no room")
        return real(*a, **kw)

    monkeypatch.setattr(W.torch, "empty", empty)
    layer, w, g = _awq_layer(2048, 1024, torch.float16, 4)
    assert len(asked) == 1 and layer.b200_expand_scratch.size() == 0
    x = torch.randn(1500, 2048, device="cuda", generator=g).to(torch.float16)
    for _ in range(3):
        out, _ = layer(x)
        assert not _lib.last_variant().endswith("expanded")
    assert len(asked) == 1
    _check(out, x, w, None)


def test_layers_on_two_streams_and_in_a_graph():
    """Layers that share the scratch, launched in turns on two streams without a synchronisation, beside replays of a
    captured one."""
    dtype, m = torch.float16, 1500
    a, wa, g = _awq_layer(4096, 2048, dtype, 5)
    b, wb, _ = _awq_layer(4096, 2048, dtype, 6)
    x = torch.randn(m, 4096, device="cuda", generator=g).to(dtype)
    ra, rb = a(x)[0].clone(), b(x)[0].clone()
    _check(ra, x, wa, None)
    _check(rb, x, wb, None)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured, _ = a(x)
    s1, s2, s3 = (torch.cuda.Stream() for _ in range(3))
    torch.cuda.synchronize()
    outs = []
    for _ in range(6):
        with torch.cuda.stream(s1):
            outs.append((a(x)[0], ra))
        with torch.cuda.stream(s2):
            outs.append((b(x)[0], rb))
        with torch.cuda.stream(s3):
            graph.replay()
    torch.cuda.synchronize()
    for o, r in outs:
        assert torch.equal(o, r)
    assert torch.equal(captured, ra)
