"""16-bit GEMM of up to 24 tokens (the small-M kernel with 16-bit operands) and just above, against float64: ragged K blocks,
channels and tokens, splits and none, 256-byte ring blocks, a bias, rows of the output that 8-byte stores do not fit.

Bound per element: one rounding to the output type (2^-8 of the result for bf16, 2^-11 for f16) and fp32 sums of K exact
products in any order, K * 2^-24 of the sum of their magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _problem(m, n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(m + 3 * n + k)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.05).to(dtype)
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    ref = x.double() @ w.double().t() + bias.double()
    return x, w, bias, ref, x.double().abs() @ w.double().abs().t() + bias.double().abs()


def _check(out, ref, mags, k):
    ulp = 2.0 ** -8 if out.dtype == torch.bfloat16 else 2.0 ** -11
    assert bool(((out.double() - ref).abs() <= ulp * ref.abs() + (k * 2.0 ** -24 + 2.0 ** -22) * mags + 2.0 ** -24).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [1, 4, 5, 16, 17, 24, 25])
@pytest.mark.parametrize("n,k", [(136, 64), (136, 72), (128, 1096), (264, 4096), (264, 4104), (24000, 1032), (20000, 2048),
                                 (20000, 2056), (24, 8192)])
def test_small(m, n, k, dtype):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.dense_kernel import gemm_16bit

    x, w, bias, ref, mags = _problem(m, n, k, dtype)
    out = gemm_16bit(x, w, bias)
    v = _lib.last_variant()
    assert v.startswith("gemm_tn kind=") and ("smallm" in v) == (m <= 24 if k > 1984 else m <= 4 and n <= 8192)
    _check(out, ref, mags, k)
    assert torch.equal(out, gemm_16bit(x, w, bias))


@pytest.mark.parametrize("m,n,k", [(4, 136, 4096), (8, 250, 4096), (20, 20000, 1024)])
@pytest.mark.parametrize("pad,shift", [(4, 0), (3, 0), (7, 1), (12, 4)])
def test_rows_that_wide_stores_do_not_fit(m, n, k, pad, shift):
    """The output as a window of a larger tensor: its neighbours keep their values."""
    from sglang_security_b200 import _lib

    x, w, bias, ref, mags = _problem(m, n, k, torch.bfloat16)
    ld = (n + 7) // 8 * 8 + pad
    whole = torch.full((m * ld + 16,), 7.0, device="cuda", dtype=torch.bfloat16)
    out = whole[shift:shift + m * ld].view(m, ld)
    rc = _lib.load().b200_gemm_16bit(x.data_ptr(), k, w.data_ptr(), k, bias.data_ptr(), out.data_ptr(), ld, m, n, k,
                                     _lib.dtype_code(torch.bfloat16), _lib.current_stream())
    _lib.check(rc, "b200_gemm_16bit")
    _check(out[:, :n], ref, mags, k)
    assert bool((out[:, n:] == 7.0).all()) and bool((whole[:shift] == 7.0).all()) and bool((whole[shift + m * ld:] == 7.0).all())
