"""The two-tile extend kernel (csrc/attn_extend_wide.cuh) at the edges of its tiles, against the oracle: one and two
query tiles per CTA (128 rows = 128 / pack tokens each), key counts around multiples of the 128-key tile, fewer and
more K / V tiles than the ring holds, both head sizes and types.

Tolerance: P and the output are rounded to 16 bits, so an element is off by at most 2^-8 (bf16) or 2^-11 (f16) of the
largest value twice over; N(0, 1) values stay below 6: 6 * 2 * 2^-8 = 0.047 and 0.006."""
import ctypes

import pytest
import torch

import harness
from oracle import scenarios

pytestmark = pytest.mark.gpu


def _run(case):
    from sglang_security_b200 import _lib

    o_ref, _, _ = harness.oracle_run(case)
    o, _, _ = harness.b200_run(case)
    assert _lib.last_variant().startswith("attn_extend_wide"), _lib.last_variant()
    n = ctypes.c_int64()
    _lib.check(_lib.load().b200_wait_timeouts(ctypes.byref(n)), "b200_wait_timeouts")
    assert n.value == 0
    st = harness.error_stats(o, o_ref)
    bound = 0.047 if case.dtype == torch.bfloat16 else 0.006
    assert st["max_abs"] <= bound and st["rel_l2"] <= (6e-3 if case.dtype == torch.bfloat16 else 1e-3), st


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 128), (8, 1, 128), (3, 1, 128), (7, 1, 64), (4, 2, 64)])
def test_tile_edges(hq, hkv, d, dtype):
    pack = next(p for p in (8, 4, 2, 1) if (hq // hkv) % p == 0)
    rows = 128 // pack                                   # tokens of a query tile
    ext = [1, rows - 1, rows, rows + 1, 2 * rows, 2 * rows + 1, 5, 1]
    longest = 1285 if d == 128 else 2941                 # makes the batch take this kernel
    total = [1, 127, 128 + rows, 129 + rows, 2 * rows, 512 + 2 * rows, longest, 641]
    _run(scenarios.make_attention_case(seed=hq * 100 + d, hq=hq, hkv=hkv, d=d, seq_lens=total, extend_lens=ext, dtype=dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("hq,hkv,d,seq,ext,splits", [
    (4, 1, 128, [3300], [40], 8),                     # one query tile, eight ranks
    (4, 1, 128, [3300, 200, 1], [64, 64, 1], 8),      # ranks without keys beside full ones
    (8, 1, 128, [1700, 900], [32, 20], 4),
    (7, 1, 64, [3073], [129], 8),                     # two query tiles, a rank with one key more
    (4, 1, 128, [1290], [90], 2),
])
def test_keys_spread_over_clusters(hq, hkv, d, seq, ext, splits, dtype):
    from sglang_security_b200 import _lib

    case = scenarios.make_attention_case(seed=sum(seq) + d, hq=hq, hkv=hkv, d=d, seq_lens=seq, extend_lens=ext, dtype=dtype)
    _run(case)
    assert f"splits={splits}" in _lib.last_variant(), _lib.last_variant()


@pytest.mark.parametrize("d", [64, 128])
def test_growing_scores_rescale(d):
    """Keys that grow along the sequence move every row's maximum again and again."""
    case = scenarios.make_attention_case(seed=5 + d, hq=4, hkv=1, d=d, seq_lens=[1500], extend_lens=[300], dtype=torch.float16)
    ramp = torch.linspace(0.1, 4.0, 1500)
    slots = case.req_to_token[case.req_pool_indices[0], :1500].long()
    case.k_cache[slots] *= ramp[:, None, None].to(case.k_cache.dtype)
    case.k_new *= ramp[1200:, None, None].to(case.k_new.dtype)
    _run(case)


@pytest.mark.parametrize("hq,hkv,d,prefix,ext,splits", [
    (4, 1, 128, [1300, 40, 0], [70, 33, 1], 2),
    (4, 1, 128, [3400, 100], [30, 65], 8),
    (8, 1, 64, [2940, 500], [40, 17], 4),
    (8, 8, 128, [900, 1000, 1100, 20, 300], [400, 270, 129, 400, 1], 1),
])
def test_every_key_visible(hq, hkv, d, prefix, ext, splits):
    """No causal mask (encoder layers): every new token sees all keys of its request, also on keys spread over ranks."""
    from sglang_security_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(sum(prefix) + d)
    total = [p + e for p, e in zip(prefix, ext)]
    slots = torch.randperm(sum(total), device="cuda", generator=g) + 1
    r2t = torch.zeros(len(ext), max(total), device="cuda", dtype=torch.int32)
    rows, at = [], 0
    for b, n in enumerate(total):
        r2t[b, :n] = slots[at:at + n].to(torch.int32)
        at += n
    kc, vc = (torch.randn(sum(total) + 1, hkv, d, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(sum(ext), hq * d, device="cuda", generator=g).to(torch.bfloat16)
    o = torch.empty_like(q)
    i32 = lambda x: torch.tensor(x, device="cuda", dtype=torch.int32)
    lens, pre = i32(ext), i32(prefix)
    starts = torch.empty_like(lens)
    lib, st = _lib.load(), _lib.current_stream()
    _lib.check(lib.b200_extend_starts(lens.data_ptr(), starts.data_ptr(), len(ext), st), "b200_extend_starts")
    idx, seq = torch.arange(len(ext), device="cuda"), torch.tensor(total, device="cuda")
    _lib.check(lib.b200_attn_extend_known(
        q.data_ptr(), q.stride(0), kc.data_ptr(), vc.data_ptr(), hkv * d, o.data_ptr(), o.stride(0), r2t.data_ptr(),
        r2t.stride(0), idx.data_ptr(), seq.data_ptr(), pre.data_ptr(), lens.data_ptr(), starts.data_ptr(), len(ext),
        max(ext), max(total), hq, hkv, d, d, d ** -0.5, 0.0, 1.0, 0, _lib.dtype_code(q.dtype), st), "b200_attn_extend_known")
    assert _lib.last_variant() == f"attn_extend_wide d={d} splits={splits}"
    row = 0
    for b, n in enumerate(total):
        at = r2t[b, :n].long()
        for h in range(hq):
            kb, vb = kc[at, h // (hq // hkv)].double(), vc[at, h // (hq // hkv)].double()
            qb = q[row:row + ext[b], h * d:(h + 1) * d].double()
            ref = (qb @ kb.t() * d ** -0.5).softmax(-1) @ vb
            got = o[row:row + ext[b], h * d:(h + 1) * d].double()
            assert (got - ref).abs().max() <= 0.047 and (got - ref).norm() <= 6e-3 * ref.norm()
        row += ext[b]


@pytest.mark.parametrize("bs", [1, 2, 255, 256, 257, 1000])
def test_start_rows(bs):
    from sglang_security_b200 import _lib

    lens = torch.randint(0, 9000, (bs,), device="cuda", dtype=torch.int32)
    starts = torch.full_like(lens, -1)
    _lib.check(_lib.load().b200_extend_starts(lens.data_ptr(), starts.data_ptr(), bs, _lib.current_stream()),
               "b200_extend_starts")
    assert torch.equal(starts.long(), lens.long().cumsum(0) - lens.long())
