"""Decode entries whose page tables name the slots that other entries are given in the same call (two positions of one
request as two entries, a fork of a request beside it, a slot named twice): all new rows are in the pool before any is read,
unless the batch says that no entry reads another's new slot (own_slots)."""
from types import SimpleNamespace

import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.attention.b200_backend import B200AttnBackend, ForwardMetadata
from sglang_security_b200.layers.radix_attention import RadixAttention
from sglang_security_b200.managers import schedule_batch as SB
from sglang_security_b200.mem_cache.memory_pool import MHATokenToKVPool, ReqToTokenPool
from sglang_security_b200.model_executor.forward_batch_info import ForwardBatch, ForwardMode

DEV = "cuda"
DTYPE_ARG = 5 + 18     # of b200_attn_decode_layer: the new rows, then q .. logit_cap


@pytest.mark.parametrize("own", [None, False, True])
def test_only_a_batch_that_says_so_has_slots_of_its_own(own, monkeypatch):
    calls = []

    class Lib:
        def __getattr__(self, name):
            return lambda *a: calls.append((name, a)) or 0

    monkeypatch.setattr(B200AttnBackend, "_new_rows", staticmethod(lambda *a: (a[1], a[2], a[6])))
    monkeypatch.setattr(_lib, "current_stream", lambda: 0)
    backend = B200AttnBackend.__new__(B200AttnBackend)
    backend.lib, backend.fused_tail, backend.forward_metadata = Lib(), False, ForwardMetadata()
    pool = MHATokenToKVPool(8, 1, torch.bfloat16, 2, 64, 1, "cpu")
    fb = SimpleNamespace(token_to_kv_pool=pool, out_cache_loc=torch.tensor([1, 2]), seq_lens=torch.tensor([1, 2]),
                         req_pool_indices=torch.tensor([1, 1]), req_to_token_pool=ReqToTokenPool(4, 8, "cpu"))
    if own is not None:            # a batch class without the field is one that does not say so
        fb.own_slots = own
    q, k, v = (torch.zeros(2, n * 64, dtype=torch.bfloat16) for n in (4, 2, 2))
    backend.forward_decode(q, k, v, RadixAttention(4, 64, 0.125, 2, 0), fb)
    assert [name for name, _ in calls] == ["b200_attn_decode_layer"]
    assert bool(calls[0][1][DTYPE_ARG] & _lib.OWN_SLOTS) == bool(own)


@pytest.mark.parametrize("rows,own", [([0, 1, 2], True), ([0, 1, 0], False)])
def test_the_scheduler_says_so_for_different_requests(rows, own, monkeypatch):
    monkeypatch.setattr(SB, "get_last_loc", lambda *a: None)
    monkeypatch.setattr(SB, "write_req_to_token_pool", lambda *a: None)
    monkeypatch.setattr(SB, "compute_position", lambda pre, ext, total: (pre, pre))
    allocator = SimpleNamespace(page_size=1, free_pages=range(8), alloc_extend=lambda *a: torch.arange(3))
    items = [SB.StepItem(SB.Req(str(i), [1, 2], req_pool_idx=r, cached_len=1), [2]) for i, r in enumerate(rows)]
    fb = SB.prepare(items, SimpleNamespace(max_context_len=9, req_to_token=None), allocator, None, None, "cpu")
    assert fb.forward_mode == ForwardMode.DECODE and fb.own_slots == own


def _decode(monkeypatch, separate, table, req, lens, locs, heads, act, pool_dtype, scales, splits, pieces):
    hq, hkv, d = heads
    g = torch.Generator(device=DEV).manual_seed(3)
    bs, slots = len(lens), int(table.max()) + 1
    rtp = ReqToTokenPool(table.shape[0], table.shape[1], DEV)
    rtp.req_to_token.copy_(table)
    kvp = MHATokenToKVPool(slots + 1, 1, pool_dtype, hkv, d, 1, DEV)
    for buf in (kvp.k_buffer[0], kvp.v_buffer[0]):
        rows = torch.randn(buf.shape, device=DEV, generator=g)
        buf.copy_(rows.to(pool_dtype).view(torch.uint8) if pool_dtype.itemsize == 1 else rows)
    # rows far from the old ones: a token that is read too early changes the output by more than its rounding
    q, k, v = (4 * torch.randn(bs, n * d, device=DEV, generator=g).to(act) for n in (hq, hkv, hkv))
    cfg = SimpleNamespace(num_attention_heads=hq, context_len=rtp.max_context_len, get_num_kv_heads=lambda tp: hkv)
    backend = B200AttnBackend(SimpleNamespace(device=DEV, req_to_token_pool=rtp, token_to_kv_pool=kvp, model_config=cfg,
                                              tp_size=1, server_args=SimpleNamespace()))
    monkeypatch.setattr(backend, "_num_splits", lambda *a: splits)
    if separate:
        monkeypatch.setattr(backend, "_new_rows", lambda *a: None)
    layer = RadixAttention(hq, d, d ** -0.5, hkv, 0)
    if scales:
        layer.k_scale_float, layer.v_scale_float = scales
    t = torch.tensor(lens, dtype=torch.int64)
    fb = ForwardBatch(forward_mode=ForwardMode.DECODE, batch_size=bs, req_pool_indices=torch.tensor(req, device=DEV),
                      seq_lens=t.to(DEV), out_cache_loc=torch.tensor(locs, device=DEV), seq_lens_sum=sum(lens), seq_lens_cpu=t,
                      req_to_token_pool=rtp, token_to_kv_pool=kvp, attn_backend=backend)
    backend.init_forward_metadata(fb)
    backend.forward_metadata.pieces = pieces
    backend.forward_metadata.workspace = backend._ensure_workspace(bs, splits, pieces)
    n0 = _lib.load().b200_launch_count()
    o = layer(q, k, v, fb)
    return o.clone(), kvp.k_buffer[0].clone(), kvp.v_buffer[0].clone(), _lib.load().b200_launch_count() - n0


def _positions(bs, n):
    """One request at lengths n, n + 1, ...: the later entries read the slots of the earlier ones."""
    table = (torch.randperm(n + bs, generator=torch.Generator().manual_seed(n)) + 1).to(torch.int32)
    return table[None].repeat(2, 1), [1] * bs, [n + i for i in range(bs)], table[n - 1:n - 1 + bs].tolist()


def _forks(bs, n):
    """Every row of the table begins with the first request's whole row, its new slot too."""
    perm = (torch.randperm(bs * (n + 8), generator=torch.Generator().manual_seed(n)) + 1).to(torch.int32).view(bs, n + 8)
    perm[:, :n] = perm[0, :n].clone()
    lens = [n] + [n + 1 + i % 7 for i in range(1, bs)]
    return perm, list(range(bs)), lens, [int(perm[b, lens[b] - 1]) for b in range(bs)]


def _twice(bs, n):
    """The new slot also stands at the start, in the middle and just before the end of its own row."""
    perm = (torch.randperm(bs * n, generator=torch.Generator().manual_seed(n)) + 1).to(torch.int32).view(bs, n)
    for at in (0, n // 2, n - 2):
        perm[:, at] = perm[:, n - 1].clone()
    return perm, list(range(bs)), [n] * bs, perm[:, n - 1].tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("heads,act,pool,scales", [
    ((32, 8, 128), torch.bfloat16, torch.bfloat16, None), ((14, 2, 64), torch.float16, torch.float16, None),
    ((48, 2, 128), torch.bfloat16, torch.bfloat16, None), ((20, 4, 128), torch.float16, torch.float8_e4m3fn, (0.5, 1.5)),
    ((14, 2, 64), torch.bfloat16, torch.float8_e5m2, None),
])
@pytest.mark.parametrize("splits,pieces", [(1, 0), (6, 0), (1, 40)])
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 19])
@pytest.mark.parametrize("tables", [_positions, _forks, _twice])
def test_same_bytes_as_a_write_before(tables, bs, splits, pieces, heads, act, pool, scales, monkeypatch):
    for n in (49, 900):
        case = tables(bs, n)
        ref = _decode(monkeypatch, True, *case, heads, act, pool, scales, splits, pieces)
        for _ in range(3):
            got = _decode(monkeypatch, False, *case, heads, act, pool, scales, splits, pieces)
            for a, b in zip(got[:3], ref[:3]):
                assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
        assert got[3] == ref[3] - (bs <= 2)


@pytest.mark.gpu
@pytest.mark.parametrize("own", [False, True])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("bs", [1, 2, 5, 40])
def test_pools_with_gaps_between_the_rows(bs, fp8, own):
    """A pool whose rows are wider than the heads, which the KV write launch does not take: the same output and rows as from a
    pool without gaps, and the gaps keep their bytes."""
    lib, hq, hkv, d, pad = _lib.load(), 8, 2, 64, 32
    g = torch.Generator(device=DEV).manual_seed(bs)
    lens = [1 + 37 * b % 200 for b in range(bs)]
    width = max(lens) + 3
    table = (torch.randperm(bs * width, device=DEV, generator=g) + 1).view(bs, width).to(torch.int32)
    seq = torch.tensor(lens, device=DEV)
    loc = table[torch.arange(bs, device=DEV), seq - 1].long()
    req = torch.arange(bs, device=DEV)
    act = torch.bfloat16
    q, k, v = (torch.randn(bs, n * d, device=DEV, generator=g).to(act) for n in (hq, hkv, hkv))
    pools = torch.randn(2, bs * width + 1, hkv * d, device=DEV, generator=g)
    pools = pools.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else pools.to(act)
    splits, out = 3, []
    ws = torch.empty(lib.b200_attn_decode_workspace_bytes(bs, hq, d, splits), dtype=torch.uint8, device=DEV)
    for gap in (0, pad):
        kv = torch.full((2, bs * width + 1, hkv * d + gap), 9, device=DEV, dtype=pools.dtype)
        kv[..., :hkv * d] = pools
        o = torch.empty(bs, hq * d, device=DEV, dtype=act)
        head = (k.data_ptr(), k.stride(0), v.data_ptr(), v.stride(0), loc.data_ptr()) + ((0,) if fp8 else ())
        mid = (q.data_ptr(), q.stride(0), kv[0].data_ptr(), kv[1].data_ptr(), kv.stride(1), o.data_ptr(), o.stride(0),
               table.data_ptr(), table.stride(0), req.data_ptr(), seq.data_ptr(), bs, hq, hkv, d, d, d ** -0.5, 0.0)
        mid += ((1.0, 1.0) if fp8 else ()) + (_lib.dtype_code(act) | (_lib.OWN_SLOTS if own else 0),)
        fn = lib.b200_attn_decode_fp8kv_layer if fp8 else lib.b200_attn_decode_layer
        rc = fn(*head, *mid, ws.data_ptr(), ws.numel(), splits, 0, None, 0, None, 0, None, _lib.current_stream())
        _lib.check(rc, "decode")
        assert bool((kv[..., hkv * d:] == 9).all())
        out.append((o, kv[..., :hkv * d].clone()))
    for a, b in zip(*out):
        assert torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))
    want = v.to(torch.float8_e4m3fn).view(torch.uint8) if fp8 else v
    assert torch.equal(out[0][1][1][loc], want)
