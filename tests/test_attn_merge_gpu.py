"""b200_attn_merge on its own: fewer and more splits than a warp's lanes and than the rows requested ahead, splits past
a short request (whose partials hold garbage), value sizes with and without 16-byte rows, few heads and
more than two an SM, against float64.
Bound: one rounding of the result plus fp32 sums over the splits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("splits,dv,hq", [(2, 128, 5), (8, 64, 5), (9, 128, 5), (33, 128, 5), (70, 192, 5), (5, 6, 5), (11, 37, 5),
                                          (9, 128, 110), (33, 64, 110), (11, 37, 110)])
def test_merge(splits, dv, hq, dtype):
    from sglang_security_b200 import _lib

    align, bs = 48, 3
    lens = torch.tensor([splits * align, 1, max(1, splits // 2) * align - 7], device="cuda", dtype=torch.int64)
    g = torch.Generator(device="cuda").manual_seed(splits + dv)
    po = torch.randn(bs, hq, splits, dv, device="cuda", generator=g)
    lse = torch.randn(bs, hq, splits, device="cuda", generator=g) * 4
    valid = []
    for b, n in enumerate(lens.tolist()):
        chunk = max(align, -(-(-(-n // splits)) // align) * align)
        valid.append(-(-n // chunk))
        po[b, :, valid[-1]:] = float("nan")
        lse[b, :, valid[-1]:] = float("nan")
    o = torch.zeros(bs, hq * dv, device="cuda", dtype=dtype)
    rc = _lib.load().b200_attn_merge(po.data_ptr(), lse.data_ptr(), o.data_ptr(), o.stride(0), lens.data_ptr(), bs, hq, dv,
                                     splits, align, _lib.dtype_code(dtype), _lib.current_stream())
    _lib.check(rc, "b200_attn_merge")
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for b in range(bs):
        w = torch.softmax(lse[b, :, :valid[b]].double() * 0.6931471805599453, -1)
        ref = torch.einsum("hs,hsd->hd", w, po[b, :, :valid[b]].double()).reshape(-1)
        mags = torch.einsum("hs,hsd->hd", w, po[b, :, :valid[b]].double().abs()).reshape(-1)
        assert bool(((o[b].double() - ref).abs() <= ulp * ref.abs() + 1e-5 * mags + 2.0 ** -24).all())
