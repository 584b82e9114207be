"""The stream GEMV with three CTAs per SM (grids that two would need a wave more for), at its edges, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [9, 15, 16])
@pytest.mark.parametrize("n,k,group", [(5120, 13824, 128), (5136, 2560, 32), (6016, 1920, 64), (27648, 5120, 128), (5120, 3072, 192)])
def test_three_ctas_per_sm(n, k, group, m, dtype):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization import w4a16_kernel as W

    g = torch.Generator(device="cuda").manual_seed(n + k + m)
    magic = 1024 if dtype == torch.float16 else 128
    q = torch.randint(-2 ** 31, 2 ** 31, (k, n // 8), device="cuda", dtype=torch.int64, generator=g).to(torch.int32)
    z = torch.randint(0, 16, (k // group, n), device="cuda", generator=g)
    scales = ((torch.rand(k // group, n, device="cuda", generator=g) + 0.5) * 0.002).to(dtype)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    out = W.w4a16_gemv_v2(x, W.gemv_stream_repack(q), (z + magic).to(dtype), scales, group, None)
    assert "ctas=3" in _lib.last_variant(), _lib.last_variant()
    shift = torch.tensor([0, 16, 4, 20, 8, 24, 12, 28], device="cuda")
    w = (((q[:, :, None] >> shift) & 15).reshape(k, n) - z.repeat_interleave(group, 0)).double()
    w *= scales.double().repeat_interleave(group, 0)
    want = x.double() @ w
    # the 16-bit result's rounding, and fp32 sums: a group's sum holds magic * sum x (1024 or 128 a weight of at most 15,
    # taken off again) of rms magic * sqrt(group), rounded about once per 16 k
    eps = torch.finfo(dtype).eps / 2
    fp32 = 2.0 ** -23 * magic * k ** 0.5 * group ** 0.5 * scales.double().amax(0)
    err = (out.double() - want).abs()
    assert (err <= want.abs() * eps + fp32).all(), err.max()
