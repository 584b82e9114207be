"""The CTA-pair GEMM (csrc/gemm_pair.cuh) at the edges of its tiles: token counts around the multiples of 32 that a
tile is cut to, one token, channel counts around 256 and not a multiple of 8 (2-byte stores), ragged K, split K over
two and three pairs, several tiles per pair; against float64.

Bound per element: one rounding to the output type (2^-8 of the result for bf16, 2^-11 for f16) and fp32 sums of K
products in any order, K * 2^-24 of the sum of their magnitudes (scaled by the epilogue)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 256, 64), (31, 257, 72), (32, 512, 4096), (33, 1000, 200), (129, 255, 320), (256, 264, 1024),
          (257, 4096, 640), (300, 4096, 8192), (70, 4096, 14336), (777, 3584, 512), (2048, 4096, 256), (1000, 24, 4096)]


def _check(out, ref, mags, k, dtype):
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    bound = ulp * ref.abs() + (k * 2.0 ** -24 + 2.0 ** -22) * mags + (2.0 ** -24 if dtype == torch.float16 else 0.0)
    assert bool(((out.double() - ref).abs() <= bound).all())


def _no_timeouts():
    from sglang_security_b200 import _lib

    n = ctypes.c_int64()
    _lib.check(_lib.load().b200_wait_timeouts(ctypes.byref(n)), "b200_wait_timeouts")
    assert n.value == 0


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_16bit(m, n, k, dtype):
    from sglang_security_b200.layers.dense_kernel import gemm_16bit

    g = torch.Generator(device="cuda").manual_seed(m * 7 + n)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(dtype)
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    ref = x.double() @ w.double().t() + bias.double()
    mags = x.double().abs() @ w.double().abs().t() + bias.double().abs()
    _check(gemm_16bit(x, w, bias), ref, mags, k, dtype)
    wide = torch.full((m, n + 5), 7.0, device="cuda", dtype=dtype)          # rows that 16-byte stores do not fit
    gemm_16bit(x, w, bias, out=wide[:, :n])
    _check(wide[:, :n], ref, mags, k, dtype)
    assert bool((wide[:, n:] == 7.0).all())
    _no_timeouts()


@pytest.mark.parametrize("m,n,k", [s for s in SHAPES if s[2] % 16 == 0 and s[0] > 32])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("per_token", [True, False])
def test_fp8(m, n, k, dtype, per_token):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_scaled_mm

    g = torch.Generator(device="cuda").manual_seed(m + n * 3)
    x = torch.randn(m, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    w = torch.randn(n, k, device="cuda", generator=g).to(torch.float8_e4m3fn)
    sa = (torch.rand(m if per_token else 1, 1, device="cuda", generator=g) + 0.5) * 0.02
    sb = torch.rand(n, 1, device="cuda", generator=g) + 0.5
    out = fp8_scaled_mm(x, w.t(), sa, sb, dtype)
    assert _lib.last_variant().startswith("gemm_tn kind=0")
    scale = sa.double() * sb.double().t()
    _check(out, (x.double() @ w.double().t()) * scale, (x.double().abs() @ w.double().abs().t()) * scale, k, dtype)
    _no_timeouts()


def test_repeatable_with_split_k():
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.dense_kernel import gemm_16bit

    x = torch.randn(300, 14336, device="cuda").to(torch.bfloat16)
    w = torch.randn(4096, 14336, device="cuda").to(torch.bfloat16)
    first = gemm_16bit(x, w)
    assert "splits=1" not in _lib.last_variant()
    for _ in range(5):
        assert torch.equal(first, gemm_16bit(x, w))


@pytest.mark.parametrize("m", [513, 600, 2048])
def test_weight_written_by_the_launch_before(m):
    """Above 512 tokens a GEMM waits for the launch before it: a weight quantised right before it is read whole."""
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_scaled_mm, sglang_per_token_quant_fp8

    n, k = 6144, 4096
    g = torch.Generator(device="cuda").manual_seed(m)
    x, sa = sglang_per_token_quant_fp8(torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16))
    for i in range(8):
        weight = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)
        torch.cuda.synchronize()
        w, sb = sglang_per_token_quant_fp8(weight)          # the allocator hands out the last round's bytes again
        out = fp8_scaled_mm(x, w.t(), sa, sb, torch.bfloat16)
        torch.cuda.synchronize()
        assert torch.equal(out, fp8_scaled_mm(x, w.t(), sa, sb, torch.bfloat16)), i
        del w, sb, out, weight
