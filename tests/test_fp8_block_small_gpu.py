"""Block-scaled FP8 GEMM of up to 32 tokens (scales requested four K blocks ahead): K slices of every length around that
distance, ragged tokens and channels, scales by token and by K block.  Bounds as in test_fp8_block_split_gpu.py."""
import pytest
import torch
from test_fp8_block_split_gpu import _check, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [1, 15, 16, 17, 32])
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
