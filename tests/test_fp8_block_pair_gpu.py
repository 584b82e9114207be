"""Block-scaled FP8 GEMM on CTA pairs (256 x 256 tiles) and on the 128-row tiles whose scales come through the same ring:
ragged tokens, channels and K, several tiles a pair, an odd number of K blocks, a bias, rows that 16-byte stores do not fit.
Bounds as in test_fp8_block_split_gpu.py."""
import pytest
import torch
from test_fp8_block_split_gpu import _check, _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n,k,form", [
    (1000, 4004, 2064, "pair"),      # a last block of 16 columns, a last tile of 164 channels, unaligned rows
    (2049, 3000, 4112, "pair"),      # a second wave, one token in the last tile, 33 blocks
    (1024, 4096, 4096, "pair"),
    (640, 6100, 2176, "pair"),       # the last tile's second half lies past N
    (520, 7176, 2064, "bn=256 tiles"), (769, 6000, 16, "bn=128"), (2048, 2112, 1152, "pair"), (900, 2112, 1152, "bn=128"),
    (3001, 4100, 48, "pair"),        # one block
    (2048, 1536, 512, "pair"),       # four blocks, which the ring of six takes whole
])
def test_forms(m, n, k, form, dtype):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.quantization.fp8_kernel import fp8_blockwise_scaled_mm

    a, b, sa, sb, bias, ref, mags = _problem(m, n, k, dtype)
    for scales in (sa, sa.t().contiguous().t()):      # by token, and by K block as the quantiser writes them
        for c in (None, bias):
            out = fp8_blockwise_scaled_mm(a, b, scales, sb, dtype, c)
            assert form in _lib.last_variant()
            _check(out, ref if c is None else ref + c.double(), mags if c is None else mags + c.double().abs(), k)
            assert torch.equal(out, fp8_blockwise_scaled_mm(a, b, scales, sb, dtype, c))
