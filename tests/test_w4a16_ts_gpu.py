"""Int4 linear with the dequantised weight in tensor memory (csrc/w4a16_ts.cu) at the edges of its tiles, splits and rings."""
import re

import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.quantization import w4a16_kernel as W


def test_takes_only_what_the_stream_layout_has():
    assert W.ts_takes(17, 144, 64, 32) and W.ts_takes(128, 4096, 4096, 128)
    for m, n, k, group in [(16, 4096, 4096, 128), (513, 4096, 4096, 128), (64, 4096, 4096, 16), (64, 4096, 4096, 96),
                           (64, 4096, 4000, 64), (64, 4104, 4096, 128), (64, 4096, 4096, 0), (512, 1 << 20, 4096, 128)]:
        assert not W.ts_takes(m, n, k, group), (m, n, k, group)


def _weight(n, k, group, dtype, g):
    magic = 1024 if dtype == torch.float16 else 128
    q = torch.randint(-2 ** 31, 2 ** 31, (k, n // 8), device="cuda", dtype=torch.int64, generator=g).to(torch.int32)
    z = torch.randint(0, 16, (k // group, n), device="cuda", generator=g)
    s = ((torch.rand(k // group, n, device="cuda", generator=g) + 0.5) * 0.002).to(dtype)
    shift = torch.tensor([0, 16, 4, 20, 8, 24, 12, 28], device="cuda")
    w = ((q[:, :, None] >> shift) & 15).reshape(k, n) - z.repeat_interleave(group, 0)
    # round16((w - z) * s): the product of 16-bit values in 32 bits is exact before its rounding
    w16 = (w.float() * s.repeat_interleave(group, 0).float()).to(dtype)
    return q, (z + magic).to(dtype), s, W.gemv_stream_repack(q), w16


# N, K, group -> (CTAs an SM, K splits) of the token counts below: a part-filled channel tile, one K block, groups of 32, a
# group over all of K, K splits of 2 .. 8 and ragged ones, more tiles than SMs (three CTAs an SM up to 64 tokens), tiles of
# up to 192 tokens (one CTA an SM)
@pytest.mark.gpu
@pytest.mark.parametrize("n,k,group,forms", [
    (16, 64, 64, {(2, 1)}),
    (144, 192, 64, {(2, 1)}),
    (272, 2048, 32, {(2, 8)}),
    (512, 1024, 1024, {(2, 4), (2, 1)}),
    (1536, 4096, 128, {(2, 8), (2, 6), (2, 4), (2, 3)}),
    (3584, 5120, 128, {(2, 5), (2, 4), (2, 2), (2, 1)}),
    (5120, 13824, 128, {(2, 6), (2, 3), (2, 1), (1, 1)}),
    (24576, 512, 128, {(3, 2), (2, 1)}),
    (19200, 576, 64, {(3, 2), (2, 1)}),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_matches_a_dense_product(n, k, group, forms, dtype):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    q, z, s, stream, w16 = _weight(n, k, group, dtype, g)
    # rounding of the result to 16 bits, 2-norm: 2^-11 / sqrt(3) (f16), 2^-8 / sqrt(3) (bf16); sums of at most 13824
    # products in 32 bits add 1e-5 at most
    limit = 1.2 * (2 ** -11 if dtype == torch.float16 else 2 ** -8) / 3 ** 0.5 + 1e-5
    taken, seen = 0, set()
    for m in (17, 31, 32, 33, 64, 65, 112, 128, 129, 192, 256, 300, 385, 512):
        if not W.ts_takes(m, n, k, group):
            continue
        taken += 1
        wide = torch.randn(m, k + 8, device="cuda", generator=g).to(dtype)
        x = wide[:, :k]                                     # rows with a stride
        bias = torch.randn(n, device="cuda", generator=g).to(dtype) if m % 2 else None
        out = W.w4a16_gemm_ts(x, stream, z, s, group, bias)
        again = W.w4a16_gemm_ts(x, stream, z, s, group, bias)
        assert _lib.last_variant().startswith("w4a16_ts"), _lib.last_variant()
        seen.add(tuple(int(re.search(rf"{name}=(\d+)", _lib.last_variant())[1]) for name in ("ctas", "splits")))
        ref = x.double() @ w16.double() + (0 if bias is None else bias.double())
        err = ((out.double() - ref).norm() / ref.norm()).item()
        assert err <= limit, (m, err, limit, _lib.last_variant())
        assert torch.equal(out, again)                      # sums of split K in rank order
    assert taken >= 6 and seen == forms
    _lib.check_waits()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_nibble_scale_and_zero_is_dequantised_exactly(dtype):
    """Unit rows of x give the weight itself: every (nibble, zero) pair under scales down to the subnormal ones."""
    n, k, group = 256, 256, 32
    g = torch.Generator(device="cuda").manual_seed(5)
    q, z, s, stream, _ = _weight(n, k, group, dtype, g)
    s = torch.exp2(-torch.randint(0, 25, s.shape, device="cuda", generator=g).float()).to(dtype) * (1 + s)
    magic = 1024 if dtype == torch.float16 else 128
    shift = torch.tensor([0, 16, 4, 20, 8, 24, 12, 28], device="cuda")
    w = ((q[:, :, None] >> shift) & 15).reshape(k, n) - (z.float() - magic).repeat_interleave(group, 0)
    want = (w * s.repeat_interleave(group, 0).float()).to(dtype)
    x = torch.eye(k, device="cuda", dtype=dtype)
    got = torch.cat([W.w4a16_gemm_ts(x[i:i + 128], stream, z, s, group) for i in range(0, k, 128)])
    assert torch.equal(got.float(), want.float())


@pytest.mark.gpu
def test_refuses_what_it_does_not_take():
    g = torch.Generator(device="cuda").manual_seed(6)
    q, z, s, stream, _ = _weight(128, 128, 64, torch.float16, g)
    x = torch.randn(513, 128, device="cuda", dtype=torch.float16)
    with pytest.raises(_lib.B200Error):
        W.w4a16_gemm_ts(x, stream, z, s, 64)
    with pytest.raises(_lib.B200Error):
        W.w4a16_gemm_ts(x[:32].to(torch.bfloat16), stream, z, s, 64)
    wide = torch.randn(32, 129, device="cuda", dtype=torch.float16)
    with pytest.raises(_lib.B200Error):
        W.w4a16_gemm_ts(wide[:, :128], stream, z, s, 64)    # rows that TMA does not take
