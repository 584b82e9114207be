"""Persistent extend attention (csrc/attn_extend_flat.cuh): ranges of keys that begin and end inside query tiles, against
float64 and against the kernels with a CTA per query tile."""
import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.radix_attention import AttentionType
from test_extend_layer_gpu import _batch

pytestmark = pytest.mark.gpu


def _exact(fb, q, k, v, hq, hkv, d, pool_dtype):
    pool, rtt = fb.token_to_kv_pool, fb.req_to_token_pool.req_to_token
    kc, vc = (b[0].view(pool_dtype) for b in (pool.k_buffer, pool.v_buffer))
    out, at = [], 0
    for b, (p, n) in enumerate(zip(fb.extend_prefix_lens_cpu, fb.extend_seq_lens_cpu)):
        idx = rtt[b, :p + n].long()
        kb, vb = (c[idx].double().transpose(0, 1).repeat_interleave(hq // hkv, 0) for c in (kc, vc))
        qb = q[at:at + n].double().view(n, hq, d).transpose(0, 1)
        s = qb @ kb.transpose(1, 2) * d ** -0.5
        s.masked_fill_(torch.arange(p + n, device="cuda")[None] > torch.arange(p, p + n, device="cuda")[:, None], float("-inf"))
        out.append((s.softmax(-1) @ vb).transpose(0, 1).reshape(n, hq * d))
        at += n
    return torch.cat(out)


# heads, head size: packs of 8, 4, 2, 1 query heads; prefix and new tokens of the requests: none new, one token, tile edges,
# a long one beside short ones, more requests than a scan step, equal ones
@pytest.mark.parametrize("hq,hkv,d", [(8, 1, 128), (8, 2, 64), (6, 3, 128), (7, 7, 64)])
@pytest.mark.parametrize("prefix,new", [
    ([0] * 5, [2100, 1, 63, 64, 65]),
    ([3000, 5, 0, 1500], [400, 257, 1, 900]),
    ([1030 + i for i in range(70)], [1 + 5 * (i % 9) for i in range(70)]),
    ([0, 1100, 0, 1100], [0, 300, 0, 640]),
    ([700] * 6, [512] * 6),
])
@pytest.mark.parametrize("pool_dtype", [torch.bfloat16, torch.float8_e4m3fn])
def test_against_float64(hq, hkv, d, prefix, new, pool_dtype, monkeypatch):
    monkeypatch.setenv("B200_EXTEND_FLAT", "1")        # also where the estimate prefers another kernel
    backend, layer, fb, (q, k, v) = _batch(len(new), prefix, new, hq, hkv, d, pool_dtype, torch.bfloat16, hq + len(new))
    backend.init_forward_metadata(fb)
    o = layer(q, k, v, fb)
    variant = _lib.last_variant()
    again = layer(q, k, v, fb)
    torch.cuda.synchronize()
    _lib.check_waits()
    assert torch.equal(o, again)                       # parts are added in the order of the keys
    assert "flat" in variant, variant
    ref = _exact(fb, q, k, v, hq, hkv, d, pool_dtype)
    # probabilities and result in bf16: 2^-9 relative each, against sums of values of order one
    assert (o.double() - ref).norm() <= 6e-3 * ref.norm() and (o.double() - ref).abs().max() <= 0.047
    monkeypatch.setenv("B200_EXTEND_FLAT", "0")
    o2 = layer(q, k, v, fb)
    assert "flat" not in _lib.last_variant()
    assert (o.double() - o2.double()).norm() <= 6e-3 * ref.norm()


def test_without_workspace_and_with_many_requests():
    """No workspace for short requests, nor for more of them than the plan's scan takes: the kernels of before."""
    n = 513
    backend, layer, fb, (q, k, v) = _batch(n, [1024] + [3] * (n - 1), [40] + [2] * (n - 1), 8, 2, 64, torch.bfloat16,
                                           torch.bfloat16, 3)
    assert _lib.load().b200_extend_layer_scratch_bytes(0, 0, n, 1064, 2, 64) == 0
    assert _lib.load().b200_extend_layer_scratch_bytes(0, 0, 1, 1000, 2, 64) == 0
    backend.init_forward_metadata(fb)
    o = layer(q, k, v, fb)
    assert "flat" not in _lib.last_variant()
    ref = _exact(fb, q, k, v, 8, 2, 64, torch.bfloat16)
    assert (o.double() - ref).norm() <= 6e-3 * ref.norm()


# what the batches above leave out: several tiles of heads a kv head (groups of 5, 7, 3, 6), f16, e5m2, pools with scales (they
# ride on the scores and on both stores of the output), no causal mask
@pytest.mark.parametrize("hq,hkv,d", [(20, 4, 128), (14, 2, 64), (12, 4, 128), (12, 2, 64)])
@pytest.mark.parametrize("act,pool_dtype,scales", [
    (torch.bfloat16, torch.bfloat16, None), (torch.float16, torch.float16, None),
    (torch.float16, torch.float8_e4m3fn, (0.5, 1.25)), (torch.bfloat16, torch.float8_e5m2, (0.75, 0.5)),
])
@pytest.mark.parametrize("causal", [True, False])
def test_head_tiles_types_scales_and_masks(hq, hkv, d, act, pool_dtype, scales, causal, monkeypatch):
    monkeypatch.setenv("B200_EXTEND_FLAT", "1")
    prefix, new = [1500, 5, 0, 2000], [400, 257, 1, 900]
    backend, layer, fb, (q, k, v) = _batch(4, prefix, new, hq, hkv, d, pool_dtype, act, hq)
    if scales:
        layer.k_scale_float, layer.v_scale_float = scales
    if not causal:
        layer.attn_type = AttentionType.ENCODER_ONLY
    backend.init_forward_metadata(fb)
    o = layer(q, k, v, fb)
    assert "flat" in _lib.last_variant(), _lib.last_variant()
    assert torch.equal(layer(q, k, v, fb), o)
    _lib.check_waits()
    pool, rtt = fb.token_to_kv_pool, fb.req_to_token_pool.req_to_token
    ks, vs = scales or (1.0, 1.0)
    kc, vc = (b[0].view(pool_dtype) for b in (pool.k_buffer, pool.v_buffer))
    at = 0
    for b, (p, n) in enumerate(zip(prefix, new)):
        idx = rtt[b, :p + n].long()
        kb, vb = (c[idx].double().transpose(0, 1).repeat_interleave(hq // hkv, 0) for c in (kc, vc))
        s = q[at:at + n].double().view(n, hq, d).transpose(0, 1) @ kb.transpose(1, 2) * (d ** -0.5 * ks)
        if causal:
            s.masked_fill_(torch.arange(p + n, device="cuda")[None] > torch.arange(p, p + n, device="cuda")[:, None], float("-inf"))
        ref = (s.softmax(-1) @ vb * vs).transpose(0, 1).reshape(n, hq * d)
        # weights and result rounded to 16 bits: 2^-9 (bf16) or 2^-12 (f16) relative each, 2-norm 1.6e-3 and 2e-4; about four
        # times that, as above
        limit = 6e-3 if act == torch.bfloat16 else 7.5e-4
        assert (o[at:at + n].double() - ref).norm() <= limit * ref.norm(), b
        at += n
