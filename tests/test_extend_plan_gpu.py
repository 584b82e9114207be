"""Which extends take the persistent kernel, and its workspace: asked once per forward, taken only where it runs."""
import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.attention import b200_backend
from sglang_security_b200.layers.radix_attention import AttentionType
from test_extend_layer_gpu import _batch

pytestmark = pytest.mark.gpu

# the estimates choose the persistent kernel: 480 CTAs of the two-tile kernel in 3.2 waves, whose last one is long (161 us
# against 184)
TURNS = ([3000] * 6, [640, 512, 100] * 2)
SHORT = ([1030], [20])                                               # and here they don't: a cluster shares the keys
WORKSPACE = 2 * 148 * (256 * 128 + 512) * 4                          # its two slots a CTA, at least


class _Counting:
    def __init__(self, lib):
        self._lib = lib
        self.asked = 0

    def __getattr__(self, name):
        if name == "b200_extend_layer_flat_bytes":
            self.asked += 1
        return getattr(self._lib, name)


def _case(lens, pool_dtype=torch.bfloat16, hq=32, hkv=8, d=128):
    backend, layer, fb, qkv = _batch(len(lens[0]), *lens, hq, hkv, d, pool_dtype, torch.bfloat16, 5)
    backend.lib = _Counting(backend.lib)
    backend.init_forward_metadata(fb)
    return backend, layer, fb, qkv


def _peak(call):
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = call()
    torch.cuda.synchronize()
    return out, torch.cuda.max_memory_allocated() - base


def test_the_choice_is_made_once_per_forward():
    backend, layer, fb, (q, k, v) = _case(TURNS)
    first = layer(q, k, v, fb)
    assert "flat" in _lib.last_variant()                             # by the estimates: nothing is forced here
    for _ in range(3):
        assert torch.equal(layer(q, k, v, fb), first)
    assert backend.lib.asked == 1
    layer.logit_cap = 30.0                                           # a layer of another form asks for itself
    layer(q, k, v, fb)
    assert "flat" not in _lib.last_variant() and backend.lib.asked == 2
    backend.init_forward_metadata(fb)                                # and so does the next forward
    layer(q, k, v, fb)
    assert backend.lib.asked == 3


@pytest.mark.parametrize("form", ["turns", "short", "capped", "non-causal", "no host lengths", "fp8 without host lengths"])
def test_workspace_only_where_the_persistent_kernel_runs(form):
    lens = SHORT if form == "short" else TURNS
    backend, layer, fb, (q, k, v) = _case(lens, torch.float8_e4m3fn if "fp8" in form else torch.bfloat16)
    if form == "capped":
        layer.logit_cap = 30.0
    elif form == "non-causal":
        layer.attn_type = AttentionType.ENCODER_ONLY
    elif "no host" in form or "without host" in form:
        fb.extend_seq_lens_cpu = fb.extend_prefix_lens_cpu = None
        backend.init_forward_metadata(fb)
    layer(q, k, v, fb)                                               # index tensors converted, kernels loaded
    out, peak = _peak(lambda: layer(q, k, v, fb))
    flat = "flat" in _lib.last_variant()
    assert flat == (form == "turns")
    dense = 2 * sum(lens[0] + lens[1]) * 8 * 128 * 2 if "fp8" in form else 0
    assert (peak >= WORKSPACE) if flat else (peak <= out.numel() * 2 + dense + (4 << 20)), peak


@pytest.mark.parametrize("pool_dtype", [torch.bfloat16, torch.float8_e5m2])
def test_without_memory_for_the_workspace_the_other_kernels_run(pool_dtype, monkeypatch):
    backend, layer, fb, (q, k, v) = _case(TURNS, pool_dtype)
    monkeypatch.setenv("B200_EXTEND_FLAT", "0")
    want = layer(q, k, v, fb)
    assert "flat" not in _lib.last_variant()
    monkeypatch.delenv("B200_EXTEND_FLAT")
    backend.init_forward_metadata(fb)
    dense = _lib.load().b200_extend_layer_dense_bytes(sum(map(sum, TURNS)), 6, 3640, 8, 128)   # the FP8 pool's copy
    empty, refused = torch.empty, []

    def no_room(*size, **kw):
        if kw.get("dtype") == torch.uint8 and size[0] >= WORKSPACE and size[0] != dense:
            refused.append(size[0])
            raise torch.cuda.OutOfMemoryError("no room")
        return empty(*size, **kw)

    monkeypatch.setattr(b200_backend.torch, "empty", no_room)
    for _ in range(2):
        got = layer(q, k, v, fb)
        assert "flat" not in _lib.last_variant()
        assert torch.equal(got, want)
    assert len(refused) == 1                                         # the next layer of the forward does not try again
    backend.init_forward_metadata(fb)
    monkeypatch.setattr(b200_backend.torch, "empty", empty)
    layer(q, k, v, fb)
    assert "flat" in _lib.last_variant()
