"""The FP8 linears' one native call: which forms take it (host logic, CPU tensors never do), and that it gives the bytes of
the separate quantiser and GEMM calls for every form that it takes."""
import pytest
import torch

from sglang_security_b200.layers.quantization import fp8_utils as U

FP8 = torch.float8_e4m3fn


def test_cpu_tensors_and_other_types_are_not_taken():
    x = torch.zeros(4, 256, dtype=torch.bfloat16)
    w, s = torch.zeros(8, 256).to(FP8), torch.ones(8)
    assert U._native_linear(x, w.t(), 256, 8, s, 1, None, False) is None
    assert U._native_linear(x.float(), w.t(), 256, 8, s, 1, None, False) is None
    with pytest.raises(Exception, match="CUDA"):
        U.apply_fp8_linear(x, w.t(), s)
    with pytest.raises(Exception, match="CUDA"):
        U.apply_w8a8_block_fp8_linear(x, w, [128, 128], torch.ones(1, 2))


class _OnDevice:
    """A CPU tensor that says it is on the GPU."""

    is_cuda = True

    def __init__(self, t):
        self._t = t

    def __getattr__(self, name):
        return getattr(self._t, name)


@pytest.mark.parametrize("host", ["weight", "scale", "bias"])
@pytest.mark.parametrize("block", [False, True])
def test_an_operand_in_host_memory_reaches_no_kernel(block, host, monkeypatch):
    def no_kernel():
        raise AssertionError("a kernel was called")

    monkeypatch.setattr(U._lib, "load", no_kernel)
    monkeypatch.setattr(U._lib, "current_stream", lambda: 0)
    x = torch.zeros(4, 256, dtype=torch.bfloat16)
    t = {"weight": torch.zeros(8, 256).to(FP8), "scale": torch.ones(1, 2) if block else torch.ones(8),
         "bias": torch.zeros(8, dtype=torch.bfloat16)}
    t["weight"] = t["weight"] if block else t["weight"].t()
    ops = {name: v if name == host else _OnDevice(v) for name, v in t.items()}
    assert U._native_linear(_OnDevice(x), ops["weight"], 256, 8, ops["scale"], 1, ops["bias"], block) is None
    mm = U.fp8_blockwise_scaled_mm if block else U.fp8_scaled_mm
    a_scale = torch.ones(4, 2 if block else 1)
    with pytest.raises(U._lib.B200Error, match="CUDA"):
        mm(_OnDevice(x.to(FP8)), ops["weight"], _OnDevice(a_scale), ops["scale"], torch.bfloat16, ops["bias"])


def test_scales_of_another_length_are_refused():
    x, w = torch.zeros(4, 256, dtype=torch.bfloat16), torch.zeros(8, 256).to(FP8)
    for n in (2, 3, 7, 9):
        with pytest.raises(ValueError, match="per-channel"):
            U.apply_fp8_linear(_OnDevice(x), w.t(), torch.ones(n))


def _both(monkeypatch, call):
    taken = []
    native = U._native_linear
    monkeypatch.setattr(U, "_native_linear", lambda *a: taken.append(native(*a)) or taken[-1])
    got = call()
    monkeypatch.setattr(U, "_native_linear", lambda *a: None)
    ref = call()
    monkeypatch.setattr(U, "_native_linear", native)
    assert got.shape == ref.shape and got.dtype == ref.dtype
    assert torch.equal(got.view(torch.int16), ref.view(torch.int16))
    return bool(taken) and taken[-1] is not None


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m", [1, 7, 40, 300, 1030])
@pytest.mark.parametrize("block", [False, True])
def test_same_bytes(m, block, dtype, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(m)
    n, k = 520, 1152
    wide = torch.randn(m, k + 64, device="cuda", generator=g).to(dtype)
    w = (torch.randn(n, k, device="cuda", generator=g) * 0.1).to(FP8)
    bias = torch.randn(n, device="cuda", generator=g).to(dtype)
    ws = torch.rand((n + 127) // 128, k // 128, device="cuda", generator=g) + 0.5
    cs = torch.rand(n, 1, device="cuda", generator=g) + 0.5

    def run(x, b, scale):
        if block:
            return U.apply_w8a8_block_fp8_linear(x, w, [128, 128], scale, bias=b)
        return U.apply_fp8_linear(x, w.t(), scale, bias=b)

    full = ws if block else cs
    for x in (wide[:, :k], wide[:, :k].contiguous(), wide[:, 8:k + 8]):
        for b in (None, bias):
            assert _both(monkeypatch, lambda: run(x, b, full))
    assert _both(monkeypatch, lambda: run(wide[:, :k].reshape(1, m, k), bias, full))
    assert _both(monkeypatch, lambda: run(wide.t().contiguous()[:k].t(), None, full))     # columns first: copied
    assert not _both(monkeypatch, lambda: run(wide[:, :k], bias.float(), full))           # a bias of another type
    assert not _both(monkeypatch, lambda: run(wide[:0, :k], None, full))                  # no tokens
    if block:
        assert not _both(monkeypatch, lambda: run(wide[:, :k], None, ws.t().contiguous().t()))
    else:
        assert _both(monkeypatch, lambda: run(wide[:, :k], None, cs[:1]))                 # one scale for all
        assert _both(monkeypatch, lambda: run(wide[:, :k], None, cs.t().contiguous()))
        assert not _both(monkeypatch, lambda: run(wide[:, :k], None, torch.cat([cs, cs], 1)[:, :1]))
    with pytest.raises(Exception, match="aligned|multiple"):
        run(wide[:, 1:k + 1], None, full)
