"""The FP8 quantisers' bytes and scales, bit by bit: every significand of a value against every significand of its
group's maximum (the group quantiser divides by a reciprocal and a remainder step), rows of every register layout of
the per-token quantiser, zeros, infinities and NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu
FP8 = torch.float8_e4m3fn


def _group_ref(x, eps=1e-10):
    f = x.float().view(x.shape[0], -1, 128)
    s = f.abs().nan_to_num(nan=0.0, posinf=float("inf")).amax(-1, keepdim=True).clamp(min=eps)
    s = s / torch.full_like(s, 448.0)      # a tensor: torch multiplies by the reciprocal of a scalar
    y = f / s
    y = torch.where(y.isnan(), torch.full_like(y, -448.0), y).clamp(-448.0, 448.0)   # max(NaN, -448) of the kernel
    return y.to(FP8).view(x.shape), s.squeeze(-1)


def _same(x, eps=1e-10):
    from sglang_security_b200.layers.quantization.fp8_kernel import per_token_group_quant_fp8

    q, s = per_token_group_quant_fp8(x, 128, eps)
    rq, rs = _group_ref(x, eps)
    assert torch.equal(s, rs)
    assert torch.equal(q.view(torch.uint8), rq.view(torch.uint8))


@pytest.mark.parametrize("dtype,bits", [(torch.bfloat16, 7), (torch.float16, 10)])
@pytest.mark.parametrize("top", [0, 3])
def test_group_quotients_exhaustively(dtype, bits, top):
    """Maximum = (1 + i / 2^bits) 2^top for all i; values (1 + j / 2^bits) 2^e for all j, e from top - 13 to top."""
    n = 1 << bits
    sig = 1.0 + torch.arange(n, device="cuda", dtype=torch.float32) / n
    vals = torch.cat([sig * 2.0 ** (top - e) for e in range(14)])
    for part in torch.arange(n, device="cuda").split(128):
        peak = sig[part] * 2.0 ** top                                     # [rows]
        rows = torch.minimum(vals.expand(len(part), -1), peak[:, None])   # none above its maximum
        pad = (-rows.shape[1]) % 127
        rows = torch.nn.functional.pad(rows, (0, pad)).view(len(part), -1, 127)
        x = torch.cat([peak[:, None, None].expand(-1, rows.shape[1], 1), rows], -1).reshape(len(part), -1)
        _same(x.to(dtype))
        _same((-x).to(dtype))


def test_group_special_values_and_sizes():
    g = torch.Generator(device="cuda").manual_seed(1)
    for m, k in ((1, 128), (3, 384), (257, 4096), (3001, 640)):
        x = (torch.randn(m, k, device="cuda", generator=g) * torch.rand(m, 1, device="cuda", generator=g) * 30).to(torch.bfloat16)
        x.view(-1)[::97] = 0
        _same(x)
    x = torch.randn(8, 256, device="cuda", generator=g).to(torch.float16)
    x[0, :128] = 0
    x[1, 5], x[2, 200], x[3, 7] = float("inf"), float("-inf"), float("nan")
    x[4] *= 1e-6
    _same(x)


@pytest.mark.parametrize("eps", [0.0, 1e-45, 1e-38, 1e-36, 2.0 ** -81, 1e-10])
def test_group_small_scales(eps):
    """Any eps is the caller's choice: scales down to the smallest subnormal (their reciprocal overflows), around the
    line from which on they are divided by, and groups whose scale is eps itself."""
    sig = 1.0 + torch.arange(128, device="cuda", dtype=torch.float32) / 128
    for top in (-132, -128, -121, -118, -100, -84, -83, -82, -81, -40, 0, 30, 120):
        peak = sig[torch.arange(0, 128, 5, device="cuda")] * 2.0 ** top
        rows = torch.cat([sig * 2.0 ** (top - e) for e in range(10)])
        rows = torch.minimum(rows.expand(len(peak), -1), peak[:, None])
        rows = torch.nn.functional.pad(rows, (0, (-rows.shape[1]) % 127)).view(len(peak), -1, 127)
        x = torch.cat([peak[:, None, None].expand(-1, rows.shape[1], 1), rows], -1).reshape(len(peak), -1).to(torch.bfloat16)
        _same(x, eps)
        _same(-x, eps)


def test_group_scale_from_eps_exhaustively():
    """Every bf16 value up to eps, of either sign, in groups whose maximum does not reach eps."""
    for eps in (1e-10, 3e-7, 1.7e-20):
        bits = torch.arange(0, 0x7f80, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
        x = bits[bits.float() <= eps]
        x = torch.cat([x, x.new_zeros((-x.numel()) % 128)]).view(-1, 128)
        _same(x, eps)
        _same(-x, eps)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [1, 7, 700])
@pytest.mark.parametrize("k", [8, 136, 896, 4096, 4104, 14336, 27648, 33000])
def test_per_token_rows(m, k, dtype):
    from sglang_security_b200.layers.quantization.fp8_kernel import sglang_per_token_quant_fp8

    g = torch.Generator(device="cuda").manual_seed(k + m)
    wide = torch.randn(m, k + 8, device="cuda", generator=g).to(dtype)
    x = wide[:, :k]                                                       # a row stride of its own
    x[0] = 0 if m > 1 else x[0]
    q, s = sglang_per_token_quant_fp8(x)
    f = x.float()
    rs = f.abs().amax(-1, keepdim=True)
    rs = rs / torch.full_like(rs, 448.0)
    inv = torch.where(rs > 0, 1.0 / rs, torch.zeros_like(rs))
    assert torch.equal(s, rs)
    assert torch.equal(q.view(torch.uint8), (f * inv).clamp(-448, 448).to(FP8).view(torch.uint8))
