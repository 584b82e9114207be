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
