"""Stream GEMV with K split over clusters whose size is no power of two (a rank then reduces ceil(128 / size) columns, the
last one fewer): unit scales and activations in {-1, 0, 1}, so every sum is a whole number below 2^24 and the result is the
exact one, rounded once."""
import pytest
import torch
from oracle import int4 as O
from test_w4a16_gpu import _prep, _rand_i32, gemv2_cfg  # noqa: F401

pytestmark = pytest.mark.gpu


def _run(m, n, k, group, dtype):
    from sglang_security_b200.layers.quantization.w4a16_kernel import gemv_stream_repack, w4a16_gemv_v2

    qweight, qzeros = _rand_i32((k, n // 8), n + m), _rand_i32((k // group, n // 8), k)
    x = torch.randint(-1, 2, (m, k), generator=torch.Generator().manual_seed(m)).to(dtype)
    bias = torch.randint(-8, 9, (n,), generator=torch.Generator().manual_seed(n)).to(dtype)
    w = O.unpack_awq_int4(qweight).float() - O.unpack_awq_int4(qzeros).float().repeat_interleave(group, 0)
    qw, zb, sc = _prep(qweight, torch.ones((k // group, n), dtype=dtype), qzeros, dtype)
    out = w4a16_gemv_v2(x.cuda(), gemv_stream_repack(qw), zb, sc, group, bias.cuda())
    exact = (x.float() @ w + bias.float()).to(dtype)
    assert torch.equal(out.cpu(), exact)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 5, 8, 13, 16])
@pytest.mark.parametrize("splits", [3, 5, 6, 7])
def test_cluster_sizes(splits, m, dtype, gemv2_cfg):  # noqa: F811
    gemv2_cfg(splits)
    _run(m, 288, 2560, 64, dtype)


@pytest.mark.parametrize("m,splits,used", [(16, 5, 8), (16, 6, 8), (16, 7, 8), (16, 3, 8), (9, 5, 8), (8, 5, 8), (1, 5, 6), (16, 1, 8)])
def test_a_slice_that_does_not_fit_grows_to_eight_ranks_at_most(m, splits, used, gemv2_cfg):  # noqa: F811
    """28672 input channels in 5 to 7 slices exceed what three CTAs share."""
    from sglang_security_b200 import _lib

    gemv2_cfg(splits)
    _run(m, 144, 28672, 128, torch.float16)
    assert f"splits={used} " in _lib.last_variant()


@pytest.mark.parametrize("units,splits", [(19, 6), (20, 6), (20, 8), (25, 6), (40, 7), (9, 8), (3, 8), (2, 7)])
def test_ranks_without_a_slice(units, splits, gemv2_cfg):  # noqa: F811
    gemv2_cfg(splits)
    for m in (1, 13):
        _run(m, 144, units * 128, 128, torch.bfloat16)


@pytest.mark.parametrize("m,n,k,splits", [(1, 7168, 4096, 6), (8, 7168, 4096, 6), (1, 896, 896, 4), (1, 28672, 1024, 2)])
def test_default_sizes(m, n, k, splits):
    """7168 channels: eight slices are more clusters than are resident at once."""
    from sglang_security_b200 import _lib

    _run(m, n, k, 128, torch.float16)
    assert f"splits={splits} " in _lib.last_variant()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 9])
@pytest.mark.parametrize("group", [32, 64, 128, 320])
@pytest.mark.parametrize("blocks", [5, 10, 15, 20, 25, 30, 35, 45])
def test_ends_of_a_slice(blocks, group, m, dtype, gemv2_cfg):  # noqa: F811
    """Slices of every length around a round of four 64-k tiles, one and two ranks (a group is whole in a slice)."""
    for splits in (1, 2):
        gemv2_cfg(splits)
        k = blocks * 64 if group != 128 else blocks * 128
        _run(m, 144, k, group, dtype)
