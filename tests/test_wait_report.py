"""A bounded wait that runs out inside a kernel is reported to the host: by the library's next launch of a kernel with
such waits, by b200_wait_error, and where the sampler hands out the tokens.  The GPU part lets one wait run out (a
barrier that nothing arrives on, a limit of a millisecond) in a process of its own, since the count of such waits is
kept for the life of the process."""
import os
import subprocess
import sys
from types import SimpleNamespace

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GREEDY = SimpleNamespace(sampling_params=SimpleNamespace(temperature=0.0), rid="r")


def test_sampler_does_not_hand_out_tokens_of_a_kernel_that_gave_up(monkeypatch):
    from sglang_security_b200 import _lib
    from sglang_security_b200.layers.sampler import Sampler

    word = [0]

    class Lib:
        def b200_wait_error(self):
            v, word[0] = word[0], 0
            return v

    monkeypatch.setattr(_lib, "load", lambda: Lib())
    logits = torch.eye(3, 8)
    sampler = Sampler("cpu")
    assert sampler(logits, [GREEDY] * 3) == [0, 1, 2]
    word[0] = 1
    with pytest.raises(_lib.B200Error, match="ran out"):
        sampler(logits, [GREEDY] * 3)
    assert sampler(logits, [GREEDY] * 3) == [0, 1, 2]      # reported once


def test_no_report_without_a_launch():
    from sglang_security_b200 import _lib, build

    build.ensure_built()
    assert _lib.load().b200_wait_error() == 0
    _lib.check_waits()


CHILD = """
import ctypes, torch
from sglang_security_b200 import _lib
from sglang_security_b200.layers.dense_kernel import gemm_16bit
lib = _lib.load()

def count():
    n = ctypes.c_int64()
    _lib.check(lib.b200_wait_timeouts(ctypes.byref(n)), "b200_wait_timeouts")
    return n.value

x = torch.randn(70, 256, device="cuda").to(torch.bfloat16)
w = torch.randn(512, 256, device="cuda").to(torch.bfloat16)
ref = gemm_16bit(x, w)
_lib.check_waits()
assert count() == 0
side = torch.cuda.Stream()                     # the count waits for streams of its own too
with torch.cuda.stream(side):
    _lib.check(lib.b200_wait_selftest(_lib.current_stream()), "b200_wait_selftest")
assert count() == 1
try:
    gemm_16bit(x, w)
    raise SystemExit("the next launch did not fail")
except _lib.B200Error as e:
    assert "ran out" in str(e), e
assert torch.equal(gemm_16bit(x, w), ref)      # reported once
_lib.check(lib.b200_wait_selftest(_lib.current_stream()), "b200_wait_selftest")
torch.cuda.synchronize()
try:
    _lib.check_waits()
    raise SystemExit("the host read did not raise")
except _lib.B200Error:
    pass
_lib.check_waits()
g = torch.cuda.CUDAGraph()                     # the word is there for captured launches too
with torch.cuda.graph(g):
    out = gemm_16bit(x, w)
g.replay()
torch.cuda.synchronize()
assert torch.equal(out, ref) and count() == 2
print("reported")
"""

CAPTURE_FIRST = """
import torch
from sglang_security_b200 import _lib
from sglang_security_b200.layers.dense_kernel import gemm_16bit
x = torch.randn(70, 256, device="cuda").to(torch.bfloat16)
w = torch.randn(512, 256, device="cuda").to(torch.bfloat16)
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):                      # the word is allocated by a launch that is being captured
    out = gemm_16bit(x, w)
g.replay()
torch.cuda.synchronize()
assert torch.equal(out, gemm_16bit(x, w))
print("reported")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("script", [CHILD, CAPTURE_FIRST], ids=["runs_out", "first_launch_captured"])
def test_a_wait_that_runs_out_is_reported(script):
    r = subprocess.run([sys.executable, "-c", script], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "reported" in r.stdout, r.stdout + r.stderr
