"""New K/V rows of an extend whose type is not that of q: they reach the pool as the pool's own write stores them."""
from types import SimpleNamespace

import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.attention.b200_backend import B200AttnBackend
from sglang_security_b200.mem_cache.memory_pool import MHATokenToKVPool, kv_write, kv_write_fp8

BF16, F16, F32, E4M3, E5M2 = torch.bfloat16, torch.float16, torch.float32, torch.float8_e4m3fn, torch.float8_e5m2


class _OnDevice:
    """A CPU tensor that says it is on the GPU: _new_rows looks at types and layouts only."""

    def __init__(self, t):
        self._t = t
        self.is_cuda = True

    def __getattr__(self, name):
        return getattr(self._t, name)


def _rows(q_dtype, k_dtype, v_dtype, pool_dtype, subclass=False):
    n, hkv, d = 3, 2, 64
    cls = type("OtherPool", (MHATokenToKVPool,), {}) if subclass else MHATokenToKVPool
    pool = cls(8, 1, pool_dtype, hkv, d, 1, "cpu")
    k, v = (torch.zeros(n, hkv * d).to(t) for t in (k_dtype, v_dtype))
    return B200AttnBackend._new_rows(q_dtype, _OnDevice(k), _OnDevice(v), pool.get_key_buffer(0), pool.get_value_buffer(0),
                                     pool, torch.arange(n), hkv, d)


def test_the_native_write_takes_rows_of_the_type_of_q_only():
    types = (BF16, F16, F32, E4M3, E5M2)
    for q in types:
        for k in types:
            for v in types:
                for pool in types:
                    taken = q in (BF16, F16) and k == v == q and pool in (q, E4M3, E5M2)
                    assert (_rows(q, k, v, pool) is not None) == taken, (q, k, v, pool)


def test_the_rows_of_a_pool_of_another_class_are_its_own_to_quantise():
    assert _rows(BF16, BF16, BF16, E4M3, subclass=True) is None
    assert _rows(BF16, BF16, BF16, BF16, subclass=True) is not None


def _extend(q_dtype, k_dtype, pool_dtype, scales=None):
    """One extend of three requests -> (output or exception, pool after it, k, v, loc, pool before)."""
    from test_extend_layer_gpu import _batch

    hq, hkv, d = 4, 2, 64
    backend, layer, fb, (q, k, v) = _batch(3, [5, 0, 70], [9, 33, 1], hq, hkv, d, pool_dtype, F32, 11)
    q, k, v = q.to(q_dtype), k.to(k_dtype), v.to(k_dtype)
    if scales:
        layer.k_scale_float, layer.v_scale_float = scales
    pool = fb.token_to_kv_pool
    before = pool.k_buffer[0].clone(), pool.v_buffer[0].clone()
    backend.init_forward_metadata(fb)
    try:
        out = layer(q, k, v, fb)
    except _lib.B200Error as e:
        out = e
    return SimpleNamespace(out=out, pool=pool, before=before, k=k, v=v, loc=fb.out_cache_loc, layer=layer, fb=fb, q=q)


def _same_bytes(a, b):
    return torch.equal(a.contiguous().view(torch.uint8), b.contiguous().view(torch.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("pool_dtype", [E4M3, E5M2])
def test_fp8_rows_are_copied_byte_for_byte(pool_dtype):
    r = _extend(BF16, pool_dtype, pool_dtype)
    kc, vc = (t.view(pool_dtype) for t in r.before)
    kv_write(r.k, r.v, kc, vc, r.loc)
    assert _same_bytes(r.pool.k_buffer[0], kc) and _same_bytes(r.pool.v_buffer[0], vc)
    # the output is that of rows which were in the pool already
    assert torch.equal(r.out, r.layer(r.q, None, None, r.fb, save_kv_cache=False))


@pytest.mark.gpu
@pytest.mark.parametrize("q_dtype,k_dtype", [(BF16, F16), (F16, BF16)])
@pytest.mark.parametrize("pool_dtype", [E4M3, E5M2])
@pytest.mark.parametrize("scales", [None, (0.5, 1.25)])
def test_rows_of_the_other_16_bit_type_are_quantised_as_what_they_are(q_dtype, k_dtype, pool_dtype, scales):
    r = _extend(q_dtype, k_dtype, pool_dtype, scales)
    kv_write_fp8(r.k, r.v, *r.before, r.loc, *(scales or (None, None)), pool_dtype)
    assert _same_bytes(r.pool.k_buffer[0], r.before[0]) and _same_bytes(r.pool.v_buffer[0], r.before[1])
    assert torch.equal(r.out, r.layer(r.q, None, None, r.fb, save_kv_cache=False))


@pytest.mark.gpu
def test_a_32_bit_pool_is_written_whole_before_its_type_is_refused():
    r = _extend(F32, F32, F32)
    assert isinstance(r.out, _lib.B200Error)
    kv_write(r.k, r.v, *r.before, r.loc)
    assert torch.equal(r.pool.k_buffer[0], r.before[0]) and torch.equal(r.pool.v_buffer[0], r.before[1])


@pytest.mark.parametrize("pool_fp8", [0, 1, 2])
def test_the_native_call_refuses_new_rows_of_other_types_before_it_writes(pool_fp8):
    """No rows and no requests: nothing would be launched, and the type is refused all the same."""
    lib, at = _lib.load(), torch.zeros(64, dtype=torch.uint8).data_ptr()

    def call(dtype):
        return lib.b200_extend_layer(_lib.EXTEND_LAYER_ARGS.pack(
            at, 128, at, at, 128, at, 128, at, 8, at, at, at, at, at, at, at, 128, 128, at, 0, 0, 0, 0, 0,
            0, 0, 0, 2, 2, 64, 64, 1, dtype, pool_fp8, 1.0, 0.0, 1.0, 1.0, 0, 0))

    assert call(_lib.BF16) == 0 and call(_lib.F16) == 0
    for dtype in (_lib.F32, _lib.FP8_E4M3, 7):
        assert call(dtype) != 0
        with pytest.raises(_lib.B200Error, match="new rows of dtype"):
            _lib.check(call(dtype), "b200_extend_layer")
