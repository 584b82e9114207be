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
