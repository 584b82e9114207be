"""Block-scaled FP8 GEMM of up to 32 tokens (scales requested four K blocks ahead): K slices of every length around that
distance, ragged tokens and channels, scales by token and by K block.  Bounds as in test_fp8_block_split_gpu.py."""
import pytest
import torch
from test_fp8_block_split_gpu import _check, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [1, 4, 5, 15, 16, 17, 32])
@pytest.mark.parametrize("n,k", [(136, 128), (136, 144), (128, 512), (264, 640), (20000, 1040), (20000, 1152), (24, 4240)])
def test_small(m, n, k, dtype):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_blockwise_scaled_mm

    a, b, sa, sb, bias, ref, mags = _problem(m, n, k, dtype)
    for scales in (sa, sa.t().contiguous().t()):
        out = fp8_blockwise_scaled_mm(a, b, scales, sb, dtype, bias)
        assert "smallm" in _lib.last_variant()
        _check(out, ref + bias.double(), mags + bias.double().abs(), k)
        assert torch.equal(out, fp8_blockwise_scaled_mm(a, b, scales, sb, dtype, bias))


@pytest.mark.parametrize("block", [True, False])
@pytest.mark.parametrize("m,n,k", [(4, 136, 4096), (8, 136, 4096), (31, 250, 2176), (64, 24000, 1024)])
@pytest.mark.parametrize("pad,shift", [(4, 0), (3, 0), (8, 1), (8, 4), (8, 2)])
def test_rows_that_wide_stores_do_not_fit(m, n, k, pad, shift, block):
    """The output as a window of a larger tensor: its neighbours keep their values."""
    from sglang_security_b200 import _lib

    a, b, sa, sb, bias, ref, mags = _problem(m, n, k, torch.bfloat16)
    ld = (n + 7) // 8 * 8 + pad
    whole = torch.full((m * ld + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[shift:shift + m * ld].view(m, ld)
    lib, dt, st = _lib.load(), _lib.dtype_code(torch.bfloat16), _lib.current_stream()
    if block:
        rc = lib.b200_fp8_gemm_block128(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), sa.data_ptr(), sa.stride(0),
                                        sa.stride(1), sb.data_ptr(), sb.stride(0), bias.data_ptr(), out.data_ptr(), ld, m, n, k,
                                        dt, st)
    else:
        ts, cs = sa[:, 0].contiguous(), sb[:, 0].repeat_interleave(128)[:n].contiguous()
        x, w = a.double() * ts.double()[:, None], b.double() * cs.double()[:, None]
        ref, mags = x @ w.t(), x.abs() @ w.abs().t()
        rc = lib.b200_fp8_gemm_rowcol(a.data_ptr(), a.stride(0), b.data_ptr(), b.stride(0), ts.data_ptr(), 1, cs.data_ptr(), 1,
                                      bias.data_ptr(), out.data_ptr(), ld, m, n, k, dt, st)
    _lib.check(rc, "fp8 gemm")
    _check(out[:, :n], ref + bias.double(), mags + bias.double().abs(), k)
    assert bool((out[:, n:] == 7.0).all()) and bool((whole[:shift] == 7.0).all()) and bool((whole[shift + m * ld:] == 7.0).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [33, 47, 48, 49])
@pytest.mark.parametrize("n,k", [(136, 4096), (6000, 1040), (520, 14336)])
def test_rowcol_up_to_48_tokens(m, n, k, dtype):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_scaled_mm

    a, b, sa, sb, bias, _, _ = _problem(m, n, k, dtype)
    ts, cs = sa[:, :1].contiguous(), sb[:, 0].repeat_interleave(128)[:n].contiguous()
    x, w = a.double() * ts.double(), b.double() * cs.double()[:, None]
    out = fp8_scaled_mm(a, b.t(), ts, cs, dtype, bias)
    assert ("smallm" in _lib.last_variant()) == (m <= 48 and k >= 4096)      # in eight slices of K
    _check(out, x @ w.t() + bias.double(), x.abs() @ w.abs().t() + bias.double().abs(), k)
    assert torch.equal(out, fp8_scaled_mm(a, b.t(), ts, cs, dtype, bias))
