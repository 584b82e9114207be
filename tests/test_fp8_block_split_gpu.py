"""Block-scaled FP8 GEMM with K split over a cluster, against float64: ragged last slices, a ragged last K block, channel
counts that 128 does not divide, a bias, and rows of the output that 16-byte stores do not fit (a row stride that 8 does
not divide, a first row that does not start on 16 bytes).

Bound per element: one rounding to the output type (2^-8 of the result for bf16, 2^-11 for f16) and fp32 sums of K scaled
products in any order, K * 2^-24 of the sum of their magnitudes."""
import re

import pytest
import torch

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


def _problem(m, n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + 3 * n + k)
    kb = (k + 127) // 128
    a = torch.randn(m, k, device="cuda", generator=g).to(FP8)
    b = torch.randn(n, k, device="cuda", generator=g).to(FP8)
    sa = torch.rand(m, kb, device="cuda", generator=g) + 0.5
    sb = (torch.rand((n + 127) // 128, kb, device="cuda", generator=g) + 0.5) * 0.01
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    x = a.double() * sa.double().repeat_interleave(128, 1)[:, :k]
    w = b.double() * sb.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    return a, b, sa, sb, bias, x @ w.t(), x.abs() @ w.abs().t()


def _check(out, ref, mags, k):
    ulp = 2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -11
    bound = ulp * ref.abs() + (k * 2.0 ** -24 + 2.0 ** -22) * mags + 2.0 ** -24
    assert bool(((out.double() - ref).abs() <= bound).all())


def _splits():
    from sglang_security_b200 import _lib

    v = _lib.last_variant()
    return int(re.fullmatch(r"fp8_block_gemm bn=128 tiles=\d+ splits=(\d+)", v).group(1))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,split", [
    (40, 200, 2176, True),       # 17 blocks of K in 5 slices: the last has one
    (129, 1000, 4224, True),     # 33 blocks
    (33, 128, 2064, True),       # a last block of 16 columns
    (300, 520, 2048, True), (64, 24, 14336, True),
    (128, 512, 1664, False),     # 13 blocks: a split saves less than it costs
])
def test_split(m, n, k, split, dtype):
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_blockwise_scaled_mm

    a, b, sa, sb, bias, ref, mags = _problem(m, n, k, dtype)
    for c in (None, bias):
        out = fp8_blockwise_scaled_mm(a, b, sa, sb, dtype, c)
        assert (_splits() > 1) == split
        _check(out, ref if c is None else ref + c.double(), mags if c is None else mags + c.double().abs(), k)
        assert torch.equal(out, fp8_blockwise_scaled_mm(a, b, sa, sb, dtype, c))


@pytest.mark.parametrize("m,n,k", [(40, 200, 2176), (40, 256, 512), (64, 136, 4096), (200, 4096, 256)])
@pytest.mark.parametrize("pad,shift", [(4, 0), (8, 1), (8, 4), (7, 3)])
def test_rows_that_wide_stores_do_not_fit(m, n, k, pad, shift):
    """The output as a window of a larger tensor: its neighbours keep their values."""
    from sglang_security_b200 import _lib

    a, b, sa, sb, bias, ref, mags = _problem(m, n, k, torch.bfloat16)
    ld = (n + 7) // 8 * 8 + pad
    whole = torch.full((m * ld + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[shift:shift + m * ld].view(m, ld)
    rc = _lib.load().b200_fp8_gemm_block128(
        a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), sa.data_ptr(), sa.stride(0), sa.stride(1), sb.data_ptr(),
        sb.stride(0), bias.data_ptr(), out.data_ptr(), ld, m, n, k, _lib.dtype_code(torch.bfloat16), _lib.current_stream())
    _lib.check(rc, "b200_fp8_gemm_block128")
    _check(out[:, :n], ref + bias.double(), mags + bias.double().abs(), k)
    assert bool((out[:, n:] == 7.0).all()) and bool((whole[:shift] == 7.0).all()) and bool((whole[shift + m * ld:] == 7.0).all())
