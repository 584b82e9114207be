"""Group quantiser for many groups (8 lanes a group) against the one for few, which tests/test_fp8_quant_exact_gpu.py checks
exhaustively: the same bytes and scales for every kind of value, in every place of a block, both scale layouts, row strides."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,k", [(1029, 8192), (300, 4096), (22000, 384), (65, 16256), (2731, 384)])
@pytest.mark.parametrize("column_major", [False, True])
@pytest.mark.parametrize("eps", [1e-10, 1e-38, 1.0])
def test_same_as_few_groups(m, k, column_major, eps, dtype):
    from sglang_security_b200.layers.quantization.fp8_kernel import per_token_group_quant_fp8

    g = torch.Generator(device="cuda").manual_seed(m + k)
    x = torch.randn(m, k + 8, device="cuda", generator=g) * torch.exp2(
        torch.randint(-40, 16, (m, 1), device="cuda", generator=g).float())
    at = torch.randint(0, m * k, (8, m), device="cuda", generator=g)
    flat = x.view(-1)
    for i, v in enumerate((float("nan"), float("inf"), -float("inf"), -0.0, 0.0, 3e38, 1e-45, 448.0)):
        flat[at[i][:max(1, m // (4 if i > 2 else 40))]] = v
    x[m // 2, :256] = 0.0
    x[m // 3, 128:384] = -0.0
    x = x.to(dtype)[:, :k]
    assert m * (k // 128) >= 8192
    q, s = per_token_group_quant_fp8(x, 128, eps, column_major_scales=column_major)
    step = max(1, 8191 // (k // 128))
    for r in range(0, m, step):
        qs, ss = per_token_group_quant_fp8(x[r:r + step], 128, eps, column_major_scales=column_major)
        assert torch.equal(q[r:r + step].view(torch.uint8), qs.view(torch.uint8))
        assert torch.equal(s[r:r + step].contiguous().view(torch.int32), ss.contiguous().view(torch.int32))
