"""The fused int4 GEMM's ring of packed words (csrc/w4a16.cu) over many laps, most of all where its slots pass from one
dequantising group to the other (a ring of three or five, two groups): a group that took an old phase of a slot for its own
dequantised old words, or the ring stood still."""
import pytest
import torch

from sglang_security_b200 import _lib
from sglang_security_b200.layers.quantization import w4a16_kernel as W
from test_w4a16_ts_gpu import _weight


def _lap_order(slots, groups, lag, wait_for_release):
    """CPU model of the ring's parities: stage i lies in slot i % slots and belongs to group i % groups.  The copies of one
    stage land late (`lag` is the stage that the memory holds back) while its followers' have landed.  -> the stage whose
    words group (lag + slots) % groups dequantises in its turn for stage lag + slots."""
    full = [0] * slots                      # completed phases of a slot: copies that have landed
    released = [0] * slots
    for i in range(lag + slots):            # every stage before the next lap of that slot, but for the late one
        if i != lag:
            full[i % slots] += 1
            released[i % slots] += 1
    slot, lap = lag % slots, (lag + slots) // slots

    def passes(done, phase):                # mbarrier.try_wait.parity: the phase of this parity is not the running one
        return done % 2 != phase % 2

    if wait_for_release and not passes(released[slot], lap - 1):
        return None                         # waits, as it should: the late stage has not been released
    return lag if passes(full[slot], lap) else None


def test_model_of_a_late_copy():
    """Without the wait for the release the group ahead takes the late slot at once; with it, it waits."""
    for slots in (3, 5):
        for lag in range(slots, 4 * slots):
            assert _lap_order(slots, 2, lag, wait_for_release=False) == lag
            assert _lap_order(slots, 2, lag, wait_for_release=True) is None


# tokens, N, K -> the instance: rings of ten and eight (one group keeps a slot), of three with swapped operands at 128 and 256
# tokens, of three and five with 128 and 256 token rows a tile; 40 to 108 stages a tile, split or not, one tile a CTA or more
CASES = [
    (24, 3584, 5120, "bm=32 swap=1"),
    (64, 3584, 5120, "bm=64 swap=1"),
    (100, 3584, 5120, "bm=128 swap=1"),
    (128, 3584, 5120, "bm=128 swap=1"),
    (160, 5120, 13824, "bm=256 swap=1"),
    (256, 5120, 13824, "bm=256 swap=1"),
    (100, 9216, 5120, "bm=128 swap=0"),
    (300, 5120, 5120, "bm=128 swap=0"),
    (100, 20480, 5120, "bm=128 swap=0"),
    (300, 10240, 5120, "bm=256 swap=0"),
    (512, 27648, 5120, "bm=256 swap=0"),
]


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,variant", CASES)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("group", [128, 32])
def test_many_laps(m, n, k, variant, dtype, group):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    q, z, s, _, w16 = _weight(n, k, group, dtype, g)
    x = torch.randn(m, k, device="cuda", generator=g).to(dtype)
    first = W.w4a16_gemm(x, q, z, s, group)
    assert variant in _lib.last_variant(), _lib.last_variant()
    ref = x.double() @ w16.double()
    # rounding of the result to 16 bits, 2-norm: 2^-11 / sqrt(3) (f16), 2^-8 / sqrt(3) (bf16); sums of 13824 products in 32
    # bits add 1e-5 at most
    limit = 1.2 * (2 ** -11 if dtype == torch.float16 else 2 ** -8) / 3 ** 0.5 + 1e-5
    assert ((first.double() - ref).norm() / ref.norm()).item() <= limit
    for _ in range(40):
        assert torch.equal(W.w4a16_gemm(x, q, z, s, group), first)
    _lib.check_waits()


def test_every_wait_of_the_kernel_has_a_limit():
    from pathlib import Path

    source = (Path(W.__file__).resolve().parents[2] / "csrc" / "w4a16.cu").read_text()
    assert "mbar_wait_bounded(" in source and "mbar_wait_counted(" in source
    assert "mbar_wait(" not in source
    assert "report_gave_up(" in source and "wait_error_arm(" in source
