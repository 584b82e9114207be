"""b200_extend_layer: the pool write, the 16-bit copy of an FP8 pool and the attention of one layer in one native call
give the bits of the three calls made one by one."""
import re
from pathlib import Path
from types import SimpleNamespace

import pytest
import torch

from sglang_security_b200 import _lib

ROOT = Path(__file__).resolve().parents[1]


def test_argument_block_matches_the_header():
    """Every field is 8 bytes, in the header's order of kinds (integer or pointer, double)."""
    text = (ROOT / "include" / "b200_hotpath.h").read_text()
    body = text[:text.index("} b200_extend_layer_args;")].rsplit("typedef struct {", 1)[1]
    kinds = ""
    for decl in re.sub(r"/\*.*?\*/", "", body, flags=re.S).split(";"):
        decl = decl.strip()
        if decl:
            kinds += ("d" if decl.startswith("double") else "i") * (decl.count(",") + 1)
            assert decl.startswith(("double", "int64_t")) or "*" in decl, decl
    fmt = re.sub(r"(\d+)([Qqd])", lambda m: m[2] * int(m[1]), _lib.EXTEND_LAYER_ARGS.format.lstrip("="))
    assert re.sub("[Qq]", "i", fmt) == kinds
    assert _lib.EXTEND_LAYER_ARGS.size == 8 * len(kinds)


def _batch(bs, prefix, new, hq, hkv, d, pool_dtype, act, seed):
    from sglang_security_b200.layers.attention.b200_backend import B200AttnBackend
    from sglang_security_b200.layers.radix_attention import RadixAttention
    from sglang_security_b200.mem_cache.memory_pool import MHATokenToKVPool, ReqToTokenPool
    from sglang_security_b200.model_executor.forward_batch_info import ForwardBatch, ForwardMode

    g = torch.Generator(device="cuda").manual_seed(seed)
    lens = [p + n for p, n in zip(prefix, new)]
    total, t = sum(lens), sum(new)
    rtp = ReqToTokenPool(bs + 1, (max(lens) + 8) // 4 * 4, "cuda")
    pool = MHATokenToKVPool(total + 16, 1, pool_dtype, hkv, d, 1, "cuda")
    for buf in (pool.k_buffer[0], pool.v_buffer[0]):
        rows = torch.randn(buf.shape, device="cuda", generator=g)
        buf.copy_(rows.to(pool_dtype).view(torch.uint8) if buf.dtype == torch.uint8 else rows)
    slots, at, loc = torch.randperm(total, device="cuda", generator=g) + 1, 0, []
    for b, n in enumerate(lens):
        rtp.req_to_token[b, :n] = slots[at:at + n].to(torch.int32)
        loc.append(slots[at + prefix[b]:at + n])
        at += n
    cfg = SimpleNamespace(num_attention_heads=hq, context_len=max(lens), get_num_kv_heads=lambda tp: hkv)
    backend = B200AttnBackend(SimpleNamespace(device="cuda", req_to_token_pool=rtp, token_to_kv_pool=pool,
                                              model_config=cfg, tp_size=1, server_args=SimpleNamespace()))
    i32 = dict(dtype=torch.int32, device="cuda")
    fb = ForwardBatch(forward_mode=ForwardMode.EXTEND, batch_size=bs,
                      req_pool_indices=torch.arange(bs, device="cuda"), seq_lens=torch.tensor(lens, device="cuda"),
                      out_cache_loc=torch.cat(loc), seq_lens_cpu=torch.tensor(lens),
                      extend_seq_lens=torch.tensor(new, **i32), extend_prefix_lens=torch.tensor(prefix, **i32),
                      extend_seq_lens_cpu=new, extend_prefix_lens_cpu=prefix, extend_num_tokens=t,
                      req_to_token_pool=rtp, token_to_kv_pool=pool, attn_backend=backend)
    qkv = torch.randn(t, (hq + 2 * hkv) * d, device="cuda", generator=g).to(act)
    return backend, RadixAttention(hq, d, d ** -0.5, hkv, 0), fb, qkv.split([hq * d, hkv * d, hkv * d], dim=-1)


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [1, 3, 300])          # 300: more requests than the threads that sum their lengths
@pytest.mark.parametrize("pool_dtype", [torch.bfloat16, torch.float8_e4m3fn, torch.float8_e5m2])
@pytest.mark.parametrize("strided", [True, False])
def test_one_call_equals_the_calls_one_by_one(bs, pool_dtype, strided):
    from sglang_security_b200.mem_cache.memory_pool import kv_write

    hq, hkv, d = 4, 2, 64
    prefix, new = [(7 * b) % 23 for b in range(bs)], [1 + (5 * b) % 19 for b in range(bs)]
    backend, layer, fb, (q, k, v) = _batch(bs, prefix, new, hq, hkv, d, pool_dtype, torch.bfloat16, bs)
    if not strided:
        k, v = k.contiguous(), v.contiguous()
    pool, fp8 = fb.token_to_kv_pool, _lib.is_fp8_kv(pool_dtype)
    if fp8:
        layer.k_scale_float, layer.v_scale_float = 0.5, 1.25
    lib, stream = _lib.load(), _lib.current_stream()
    assert stream == torch.cuda.current_stream().cuda_stream
    kb, vb = pool.k_buffer[0].clone(), pool.v_buffer[0].clone()
    backend.init_forward_metadata(fb)
    o = layer(q, k, v, fb)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        assert _lib.current_stream() == side.cuda_stream
    # one by one, on the pool as it was
    got = pool.k_buffer[0].clone(), pool.v_buffer[0].clone()
    pool.k_buffer[0].copy_(kb)
    pool.v_buffer[0].copy_(vb)
    if fp8:
        pool.set_kv_buffer(layer, fb.out_cache_loc, k, v, 0.5, 1.25)
    else:
        kv_write(k, v, pool.k_buffer[0], pool.v_buffer[0], fb.out_cache_loc)
    assert torch.equal(pool.k_buffer[0].view(torch.uint8), got[0].view(torch.uint8))
    assert torch.equal(pool.v_buffer[0].view(torch.uint8), got[1].view(torch.uint8))
    kc, vc, rtt, idx = pool.k_buffer[0], pool.v_buffer[0], fb.req_to_token_pool.req_to_token, fb.req_pool_indices
    total, longest, scale, out_scale = int(fb.seq_lens.sum()), int(fb.seq_lens.max()), layer.scaling, 1.0
    if fp8:
        indptr = torch.zeros(bs + 1, dtype=torch.int32, device="cuda")
        indptr[1:] = fb.seq_lens.cumsum(0)
        k16 = torch.empty(total, hkv * d, dtype=q.dtype, device="cuda")
        v16, dense = torch.empty_like(k16), torch.empty(bs, (longest + 3) // 4 * 4, dtype=torch.int32, device="cuda")
        _lib.check(lib.b200_kv_dequant_gather(
            kc.data_ptr(), vc.data_ptr(), hkv * d, rtt.data_ptr(), rtt.stride(0), idx.data_ptr(), fb.seq_lens.data_ptr(),
            indptr.data_ptr(), k16.data_ptr(), v16.data_ptr(), dense.data_ptr(), dense.stride(0), bs, longest,
            _lib.kv_dtype_code(q.dtype, pool_dtype), stream), "dequant")
        kc, vc, rtt, idx, scale, out_scale = k16, v16, dense, torch.arange(bs, device="cuda"), scale * 0.5, 1.25
    want = torch.empty_like(o)
    _lib.check(lib.b200_attn_extend_known(
        q.data_ptr(), q.stride(0), kc.data_ptr(), vc.data_ptr(), hkv * d, want.data_ptr(), want.stride(0), rtt.data_ptr(),
        rtt.stride(0), idx.data_ptr(), fb.seq_lens.data_ptr(), fb.extend_prefix_lens.data_ptr(),
        fb.extend_seq_lens.data_ptr(), backend.forward_metadata.qo_indptr.data_ptr(), bs, max(new), longest, hq, hkv, d, d,
        scale, 0.0, out_scale, 1, _lib.dtype_code(q.dtype), stream), "extend")
    assert torch.equal(o.view(torch.int16), want.view(torch.int16))
    # rows that are in the pool already, and rows of another layout, go the same way
    assert torch.equal(layer(q, k, v, fb, save_kv_cache=False), o)
    wide = torch.zeros(k.shape[0], hkv, 2 * d, dtype=k.dtype, device="cuda")
    wide[:, :, :d] = k.reshape(-1, hkv, d)
    assert torch.equal(backend.forward(q, wide[:, :, :d], v.reshape(-1, hkv, d), layer, fb), o)


@pytest.mark.gpu
def test_refused_as_before():
    backend, layer, fb, (q, k, v) = _batch(2, [3, 4], [2, 2], 4, 2, 64, torch.float16, torch.bfloat16, 1)
    backend.init_forward_metadata(fb)
    with pytest.raises(_lib.B200Error):      # bf16 rows, f16 pool
        layer(q, k, v, fb)
    backend, layer, fb, (q, k, v) = _batch(2, [3, 4], [2, 2], 4, 2, 64, torch.float8_e4m3fn, torch.bfloat16, 1)
    layer.k_scale_float = 0.5                # one scale without the other
    backend.init_forward_metadata(fb)
    with pytest.raises(_lib.B200Error):
        layer(q, k, v, fb)
    backend, layer, fb, (q, k, v) = _batch(2, [3, 4], [2, 2], 4, 2, 64, torch.bfloat16, torch.bfloat16, 1)
    backend.init_forward_metadata(fb)
    with pytest.raises(_lib.B200Error):      # rows of half the cache's width
        backend.forward(q, k[:, :64], v[:, :64], layer, fb)
