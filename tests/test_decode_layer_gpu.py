"""Decode whose split kernel stores the new K/V rows itself: output and pools are the same bytes as with a KV write of its
own before it, for page tables in any order, splits, several head tiles, entries without tokens, FP8 pools with and without
scales, and rows that 16-byte loads do not fit (those are written by a launch before)."""
from types import SimpleNamespace

import pytest
import torch

from sglang_security_b200.layers.attention.b200_backend import B200AttnBackend
from sglang_security_b200.layers.radix_attention import RadixAttention
from sglang_security_b200.mem_cache.memory_pool import MHATokenToKVPool, ReqToTokenPool
from sglang_security_b200.model_executor.forward_batch_info import ForwardBatch, ForwardMode

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _run(monkeypatch, own, heads, act, pool_dtype, lens, splits, scales, pad, pieces=0, width=9, cap=0.0, replay=None,
         replay_eager=False):
    """replay: lengths (none longer) that a graph, captured with `lens`, is replayed with, or a direct call made."""
    from sglang_security_b200 import _lib

    hq, hkv, d = heads
    g = torch.Generator(device=DEV).manual_seed(7)
    bs, total = len(lens), sum(lens) + len(lens)
    rtp = ReqToTokenPool(bs + 1, max(lens) + width, DEV)
    kvp = MHATokenToKVPool(total + 16, 1, pool_dtype, hkv, d, 1, DEV)
    for buf in (kvp.k_buffer[0], kvp.v_buffer[0]):
        rows = torch.randn(buf.shape, device=DEV, generator=g)
        buf.copy_(rows.to(pool_dtype).view(torch.uint8) if pool_dtype.itemsize == 1 else rows)
    slots = torch.randperm(total, device=DEV, generator=g) + 1
    loc, at = [], 0
    for b, n in enumerate(lens):
        rtp.req_to_token[b, :n] = slots[at:at + n].to(torch.int32)
        loc.append(slots[at + max(n - 1, 0)])          # an entry without tokens has a slot too
        at += n + 1
    width = (hq + 2 * hkv) * d
    qkv = torch.randn(bs, width + pad, device=DEV, generator=g).to(act)[:, :width]
    q, k, v = qkv.split([hq * d, hkv * d, hkv * d], dim=-1)
    q = q.contiguous()
    cfg = SimpleNamespace(num_attention_heads=hq, context_len=rtp.max_context_len, get_num_kv_heads=lambda tp: hkv)
    backend = B200AttnBackend(SimpleNamespace(device=DEV, req_to_token_pool=rtp, token_to_kv_pool=kvp, model_config=cfg,
                                              tp_size=1, server_args=SimpleNamespace(triton_attention_num_kv_splits=splits)))
    monkeypatch.setattr(backend, "_num_splits", lambda *a: splits)
    if not own:
        monkeypatch.setattr(backend, "_new_rows", lambda *a: None)
    layer = RadixAttention(hq, d, d ** -0.5, hkv, 0, logit_cap=cap)
    if scales:
        layer.k_scale_float, layer.v_scale_float = scales
    t = torch.tensor(lens, dtype=torch.int64)
    fb = ForwardBatch(forward_mode=ForwardMode.DECODE, batch_size=bs,
                      req_pool_indices=torch.arange(bs, dtype=torch.int64, device=DEV), seq_lens=t.to(DEV),
                      out_cache_loc=torch.stack(loc), seq_lens_sum=sum(lens), seq_lens_cpu=t, req_to_token_pool=rtp,
                      token_to_kv_pool=kvp, attn_backend=backend, own_slots=True)
    backend.init_forward_metadata(fb)
    if pieces:
        backend.forward_metadata.pieces = pieces
        backend.forward_metadata.workspace = backend._ensure_workspace(bs, splits, pieces)
        backend.forward_metadata.workspace.fill_(0xff)       # NaN in every partial row
    if replay:
        pools = [buf.clone() for buf in (kvp.k_buffer[0], kvp.v_buffer[0])]
        layer(q, k, v, fb)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            o = layer(q, k, v, fb)
        lens = replay
        fb.seq_lens.copy_(torch.tensor(lens))
        fb.out_cache_loc.copy_(rtp.req_to_token[torch.arange(bs), (fb.seq_lens.cpu() - 1).clamp(min=0)])
        for buf, old in zip((kvp.k_buffer[0], kvp.v_buffer[0]), pools):
            buf.copy_(old)
        if pieces:
            backend.forward_metadata.workspace.fill_(0xff)
        if replay_eager:
            o = layer(q, k, v, fb)
        else:
            graph.replay()
        torch.cuda.synchronize()
    n0 = _lib.load().b200_launch_count()
    if not replay:
        o = layer(q, k, v, fb)
    launches = _lib.load().b200_launch_count() - n0
    live = torch.tensor([n > 0 for n in lens], device=DEV)
    return o[live].clone(), kvp.k_buffer[0].clone(), kvp.v_buffer[0].clone(), launches


@pytest.mark.parametrize("splits", [1, 5])
@pytest.mark.parametrize("heads,act,pool,scales,pad", [
    ((32, 8, 128), torch.bfloat16, torch.bfloat16, None, 0),
    ((14, 2, 64), torch.float16, torch.float16, None, 8),
    ((48, 2, 128), torch.bfloat16, torch.bfloat16, None, 0),             # three head tiles of a kv head
    ((8, 2, 64), torch.bfloat16, torch.bfloat16, None, 3),               # rows that do not start on 16 bytes
    ((32, 8, 128), torch.bfloat16, torch.float8_e4m3fn, None, 0),
    ((20, 4, 128), torch.float16, torch.float8_e4m3fn, (0.5, 1.5), 0),
    ((14, 2, 64), torch.bfloat16, torch.float8_e5m2, (0.25, 2.0), 16),
    ((40, 2, 64), torch.bfloat16, torch.float8_e4m3fn, None, 0),
])
def test_same_bytes_as_a_write_before(heads, act, pool, scales, pad, splits, monkeypatch):
    lens = [1, 0, 17, 48, 49, 300, 96, 97, 3]
    got = _run(monkeypatch, True, heads, act, pool, lens, splits, scales, pad)
    ref = _run(monkeypatch, False, heads, act, pool, lens, splits, scales, pad)
    for a, b in zip(got[:3], ref[:3]):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert got[3] == ref[3] - (pad != 3)


@pytest.mark.parametrize("heads,act,pool,scales", [
    ((32, 8, 128), torch.bfloat16, torch.bfloat16, None), ((14, 2, 64), torch.float16, torch.float16, None),
    ((48, 2, 128), torch.bfloat16, torch.bfloat16, None), ((20, 4, 128), torch.float16, torch.float8_e4m3fn, (0.5, 1.5)),
    ((40, 2, 64), torch.bfloat16, torch.float8_e4m3fn, None), ((8, 2, 64), torch.bfloat16, torch.float8_e5m2, None),
])
@pytest.mark.parametrize("lens,pieces", [
    ([1, 0, 17, 48, 49, 300, 96, 97, 3], 9),                     # a piece a request at most
    ([1, 0, 17, 48, 49, 300, 96, 97, 3], 14),
    ([0, 5000, 1, 0, 700, 0], 40),                               # a request in many pieces; the last entries are empty
    ([7 + 37 * i % 911 for i in range(128)], 148),               # the largest batch
    ([2000, 96, 96], 64),                                        # more pieces than tiles need
    ([33], 1),
])
def test_pieces_of_equal_length(heads, act, pool, scales, lens, pieces, monkeypatch):
    """Against one split a request, which sums the same terms in another order: the probabilities are rounded once to 16
    bits (f16 or bf16: 2^-9 of each) and the output once, so the outputs differ by 2^-8 in the 2-norm and no element by more
    than that of the largest |v| (6 at most here, times the scale)."""
    got = _run(monkeypatch, True, heads, act, pool, lens, 1, scales, 0, pieces)
    ref = _run(monkeypatch, True, heads, act, pool, lens, 1, scales, 0)
    for a, b in zip(got[1:3], ref[1:3]):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    a, b = got[0].double(), ref[0].double()
    assert bool(a.isfinite().all())
    assert (a - b).norm() <= 2.0 ** -8 * b.norm()
    assert (a - b).abs().max() <= 2.0 ** -8 * 6 * (scales[1] if scales else 1.0)


FORMS = [((32, 8, 128), torch.bfloat16, torch.bfloat16, None), ((14, 2, 64), torch.float16, torch.float16, None),
         ((48, 2, 128), torch.bfloat16, torch.bfloat16, None), ((20, 4, 128), torch.float16, torch.float8_e4m3fn, (0.5, 1.5)),
         ((8, 2, 64), torch.bfloat16, torch.float8_e5m2, None)]
UNEQUAL = [3000, 0, 17, 1448, 649, 2300, 96, 1197, 1]


def _same(a, b):
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(x.view(torch.uint8), y.view(torch.uint8))


@pytest.mark.parametrize("heads,act,pool,scales", FORMS)
@pytest.mark.parametrize("splits,pieces", [(3, 0), (1, 24), (1, 60)])
def test_page_tables_that_take_wide_loads(heads, act, pool, scales, splits, pieces, monkeypatch):
    """Rows of a multiple of four entries: 16-byte loads, and from five tiles a warp on the step without checks.  The same
    bytes as from rows whose entries are loaded and checked one by one; new rows stored by the kernel, or before it."""
    for own in (True, False):
        wide = _run(monkeypatch, own, heads, act, pool, UNEQUAL, splits, scales, 0, pieces, width=12)
        _same(wide, _run(monkeypatch, own, heads, act, pool, UNEQUAL, splits, scales, 0, pieces, width=9))


@pytest.mark.parametrize("heads,act,pool,scales", FORMS[:3])         # FP8 pools refuse such rows
@pytest.mark.parametrize("pieces", [14, 40])
def test_pieces_with_rows_that_do_not_start_on_16_bytes(heads, act, pool, scales, pieces, monkeypatch):
    got = _run(monkeypatch, True, heads, act, pool, UNEQUAL, 1, scales, 3, pieces, width=12)
    _same(got, _run(monkeypatch, False, heads, act, pool, UNEQUAL, 1, scales, 3, pieces, width=12))


@pytest.mark.parametrize("heads,act,pool,scales", FORMS)
def test_pieces_with_a_logit_cap(heads, act, pool, scales, monkeypatch):
    """Bounds as above; the cap's own arithmetic is the same in both."""
    got = _run(monkeypatch, True, heads, act, pool, UNEQUAL, 1, scales, 0, 40, width=12, cap=5.0)
    ref = _run(monkeypatch, True, heads, act, pool, UNEQUAL, 1, scales, 0, width=12, cap=5.0)
    plain = _run(monkeypatch, True, heads, act, pool, UNEQUAL, 1, scales, 0, 40, width=12)
    a, b = got[0].double(), ref[0].double()
    assert (a - b).norm() <= 2.0 ** -8 * b.norm() and (a - b).abs().max() <= 2.0 ** -8 * 6 * (scales[1] if scales else 1.0)
    assert (a - plain[0].double()).norm() > 2.0 ** -6 * b.norm()          # the cap does something


@pytest.mark.parametrize("heads,act,pool,scales", FORMS)
@pytest.mark.parametrize("width", [9, 12])
@pytest.mark.parametrize("lens", [[1, 2999, 0, 700, 5, 2300, 0, 33, 1100], [1] * 9, [0, 0, 3000, 0, 0, 0, 0, 0, 0],
                                  [2999] * 9])
def test_a_captured_launch_follows_the_lengths(lens, width, heads, act, pool, scales, monkeypatch):
    """The plan is made from the lengths on the device: a graph captured with other lengths gives the bytes of a direct call."""
    run = lambda eager: _run(monkeypatch, True, heads, act, pool, [3000] * 9, 1, scales, 0, 40, width=width,  # noqa: E731
                             replay=lens, replay_eager=eager)
    _same(run(False), run(True))


def test_rule_of_the_pieces():
    from sglang_security_b200 import _lib

    lib = _lib.load()
    f = lambda bs, total, longest, hkv=8, group=4: lib.b200_attn_decode_pieces(bs, hkv, group, total, longest, 148)  # noqa: E731
    assert f(27, 27 * 3750, 6000) == 74 and f(16, 20000, 2000) == 74
    assert f(27, 27 * 4096, 4096) == 0                           # equal requests
    assert f(64, 64 * 1000, 1500) == 0 and f(4, 10000, 4000) == 0 and f(8, 10000, 2000) == 0 and f(129, 10 ** 6, 10 ** 5) == 0
    d64 = lambda bs, total, longest: lib.b200_attn_decode_pieces_for(bs, 2, 7, 64, total, longest, 148)  # noqa: E731
    assert d64(34, 80826, 3663) == 0 and d64(23, 176120, 15900) == 296         # splits even out the first by themselves
    assert f(40, 40 * 1915, 3064, 4, 5) == 148 and f(27, 27 * 3750, 6000, 2, 24) == 148
