"""CPU tests of the C-ABI boundary: the library builds for sm_100a, loads, and exports every
symbol include/b200_hotpath.h declares.  No compute call is made (no GPU here)."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib_path():
    from sglang_security_b200 import build

    return build.build()


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "b200_hotpath.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(b200_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported(lib_path):
    lib = ctypes.CDLL(str(lib_path))
    declared = _declared_symbols()
    assert len(declared) >= 8
    missing = [s for s in declared if not hasattr(lib, s)]
    assert not missing, f"declared in the header but not exported: {missing}"


def test_python_binding_covers_header(lib_path):
    from sglang_security_b200 import _lib

    assert sorted(_lib.exported_symbols()) == _declared_symbols()
    lib = _lib.load()
    assert lib.b200_version() >= 1
    assert lib.b200_launch_count() >= 0


def test_host_side_helpers_need_no_gpu(lib_path):
    from sglang_security_b200 import _lib

    lib = _lib.load()
    # pure host functions: workspace sizing and the split heuristic
    assert lib.b200_attn_decode_workspace_bytes(64, 32, 128, 1) == 0
    assert lib.b200_attn_decode_workspace_bytes(64, 32, 128, 4) == 64 * 32 * 4 * (128 + 1) * 4
    s = lib.b200_attn_decode_num_splits(64, 8, 4, 128, 4096, 148)
    assert s == 1   # 512 CTAs fit the 592 resident slots: one balanced wave, no merge
    # per-rank head counts of TP 2 / 4 / 8: the largest split count that still fits one wave
    assert lib.b200_attn_decode_num_splits(64, 4, 4, 128, 4096, 148) == 2
    assert lib.b200_attn_decode_num_splits(64, 2, 4, 128, 4096, 148) == 4
    assert lib.b200_attn_decode_num_splits(64, 1, 4, 128, 4096, 148) == 9
    assert lib.b200_attn_decode_num_splits(1, 8, 4, 128, 100, 148) == 1
    assert lib.b200_attn_decode_split_align(128, 4) == 48  # 3 warps x 16-token tiles


@pytest.mark.parametrize("bs,hkv,group,d,avg,longest,splits", [
    # short requests are not split, few ones from some 300 tokens on, many from some 600 on
    (1, 8, 4, 128, 128, 0, 1), (1, 8, 4, 128, 300, 0, 4), (1, 8, 4, 128, 384, 0, 8), (16, 8, 4, 128, 384, 0, 1),
    (16, 8, 4, 128, 512, 0, 1), (16, 8, 4, 128, 700, 0, 4), (5, 8, 4, 128, 300, 400, 5),
    # few requests: splits grow with the longest, up to 64
    (1, 8, 4, 128, 1500, 0, 16), (1, 8, 4, 128, 4096, 0, 18), (1, 2, 4, 128, 16384, 0, 57), (1, 8, 4, 128, 131072, 0, 64),
    (1, 8, 4, 128, 1000000, 0, 64), (2, 2, 7, 64, 1000, 4096, 29),
    # one full wave of CTAs
    (5, 8, 4, 128, 8192, 0, 14), (40, 4, 5, 128, 2048, 0, 3), (64, 8, 4, 128, 4096, 0, 1), (64, 8, 4, 128, 131072, 0, 1),
    # a wave that would be half empty: oversubscribed where the requests are long enough
    (40, 8, 4, 128, 1024, 0, 1), (40, 8, 4, 128, 3000, 0, 3),
    # unequal requests with few splits: twice the slots
    (64, 8, 4, 128, 2500, 4096, 3), (27, 8, 4, 128, 3600, 6000, 6), (64, 8, 4, 128, 1000, 1100, 1),
])
def test_split_rule(lib_path, bs, hkv, group, d, avg, longest, splits):
    from sglang_security_b200 import _lib

    lib = _lib.load()
    if longest == 0:
        assert lib.b200_attn_decode_num_splits(bs, hkv, group, d, avg, 148) == splits
        longest = avg
    assert lib.b200_attn_decode_num_splits_ragged(bs, hkv, group, d, avg, longest, 148) == splits


def test_split_rule_stays_within_the_workspace_of_graphs(lib_path):
    from sglang_security_b200 import _lib

    lib = _lib.load()
    for bs in (1, 3, 17, 64, 300, 5000):
        for hkv in (1, 2, 8, 32):
            for avg in (1, 47, 500, 3000, 70000, 1 << 22):
                for longest in (avg, 3 * avg, 1 << 23):
                    assert 1 <= lib.b200_attn_decode_num_splits_ragged(bs, hkv, 4, 128, avg, longest, 148) <= 64


def test_noalloc_decode_rejects_oversize_requests_before_touching_the_gpu(lib_path):
    """b200_attn_decode_noalloc: the size check against the built-in 8 MiB scratch comes before any
    CUDA call, so it can be exercised here (pointers are never dereferenced)."""
    from sglang_security_b200 import _lib

    lib = _lib.load()
    assert lib.b200_attn_decode_workspace_bytes(64, 32, 128, 8) > (8 << 20)
    fake = 0x1000
    rc = lib.b200_attn_decode_noalloc(fake, 4096, fake, fake, 1024, fake, 4096, fake, 64, fake, fake,
                                      64, 32, 8, 128, 128, 0.088, 0.0, _lib.BF16, 8, None)
    assert rc == 1
    msg = lib.b200_last_error().decode()
    assert "8388608" in msg and "scratch" in msg
    assert lib.b200_attn_decode_noalloc(fake, 4096, fake, fake, 1024, fake, 4096, fake, 64, fake, fake,
                                        0, 32, 8, 128, 128, 0.088, 0.0, _lib.BF16, 8, None) == 0  # empty batch


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
    from sglang_security_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "_LIB_PATH", tmp_path / "nope.so")
    with pytest.raises(_lib.B200Error):
        _lib.load()
