"""The C-ABI library builds, loads without a GPU and exports what include/nq_fp8.h declares."""
import ctypes
import os
import re

import torch

from conftest import ROOT


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "nq_fp8.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(nq_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_are_exported_and_bound(built_library):
    from nano_qwen_b200 import _cabi
    names = declared_symbols()
    assert "nq_fp8_gemm_bs128" in names and "nq_act_quant_e4m3_g128" in names and len(names) >= 12
    handle = ctypes.CDLL(built_library)
    for name in names:
        assert hasattr(handle, name), f"{name} declared in include/nq_fp8.h but not exported"
    assert sorted(_cabi.SIGNATURES) == names          # the ctypes binding covers exactly the header


def test_version_and_status_strings(built_library):
    from nano_qwen_b200 import _cabi
    lib = _cabi.lib()
    assert lib.nq_version() == 100
    assert lib.nq_status_string(0) == b"ok"
    assert b"wait" in lib.nq_status_string(-5)
    assert lib.nq_fp8_gemm_workspace_bytes(16, 4096, 4096) == 0
    assert lib.nq_launch_count() >= 0


def test_auto_dispatch_by_rounds_of_tiles(built_library):
    """Both sides of each line of the rule, with 148 SMs: the choice needs no GPU."""
    from nano_qwen_b200 import _cabi
    lib = _cabi.lib()
    W, T128, T256, PAIR = _cabi.ALGO_WEIGHT_LANE, _cabi.ALGO_TOKEN_LANE_128, _cabi.ALGO_TOKEN_LANE_256, _cabi.ALGO_TOKEN_PAIR
    for m, n, split, want in [
            (1, 4096, 0, W), (64, 24576, 0, W), (65, 24576, 0, T256),         # 192 tiles of 128 x 128 and 96 of 128 x 256
            (128, 148 * 128, 0, T128), (128, 149 * 128, 0, T256),             # one round of 128-wide tiles, and one tile more
            (4096, 128, 0, T128), (4096, 129, 0, T128),
            (520, 4104, 0, PAIR), (520, 4104, 1, PAIR), (520, 4104, 2, T256), # a K split goes to a kernel that can split
            (777, 6144, 0, T128), (777, 24576, 0, T256), (1281, 4088, 0, T128), (2047, 1000, 0, T128),
            (2047, 4736, 0, T128), (2048, 4736, 0, PAIR), (2048, 4736, 4, PAIR), (8192, 6144, 0, PAIR)]:
        assert lib.nq_gemm_auto_algo(m, n, split, 148) == want, (m, n, split)
    assert lib.nq_gemm_auto_algo(0, 128, 0, 148) == lib.nq_gemm_auto_algo(1, 128, 0, 0) == -1


def test_auto_dispatch_counts_rounds_without_the_sms_held_back(built_library):
    """140 tiles of 128 x 128 are one round of 148 SMs and two of 128, where 70 tiles of 128 x 256 are one."""
    from nano_qwen_b200 import _cabi
    lib = _cabi.lib()
    old = lib.nq_set_sm_reserve(0)
    try:
        assert lib.nq_gemm_auto_algo(512, 35 * 128, 2, 148) == _cabi.ALGO_TOKEN_LANE_128
        assert lib.nq_gemm_auto_algo(2048, 34 * 128, 0, 148) == _cabi.ALGO_TOKEN_PAIR            # 8 x 17 tiles: two rounds
        lib.nq_set_sm_reserve(20)
        assert lib.nq_gemm_auto_algo(512, 35 * 128, 2, 148) == _cabi.ALGO_TOKEN_LANE_256
        assert lib.nq_gemm_auto_algo(2048, 34 * 128, 0, 148) == _cabi.ALGO_TOKEN_PAIR
        lib.nq_set_sm_reserve(1000)                                           # at least half of the SMs stay
        assert lib.nq_gemm_auto_algo(512, 18 * 128, 2, 148) == _cabi.ALGO_TOKEN_LANE_128         # 72 tiles, 74 CTAs
        assert lib.nq_gemm_auto_algo(512, 19 * 128, 2, 148) == _cabi.ALGO_TOKEN_LANE_256
    finally:
        lib.nq_set_sm_reserve(old)


def test_no_cpu_fallback():
    """Without a CUDA device every compute entry refuses loudly instead of computing elsewhere."""
    import pytest
    from nano_qwen_b200 import _cabi, ops
    x = torch.zeros(4, 128, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        ops.act_quant(x)
    with pytest.raises(RuntimeError, match="no CPU fallback"):
        ops.fp8_linear(x, torch.zeros(128, 128).to(torch.float8_e4m3fn), torch.ones(1, 1))
    if not torch.cuda.is_available():
        with pytest.raises(_cabi.NqError):
            ops.init()


def test_stream_handle_without_torchs_private_names(monkeypatch):
    """The raw-handle query is a shortcut: a torch without it is asked through its public interface."""
    import types
    from nano_qwen_b200 import ops
    monkeypatch.setattr(ops, "_raw_stream", lambda device: 1000 + device, raising=False)
    monkeypatch.setattr(ops, "_device", lambda: 3, raising=False)
    assert ops._stream() == 1003
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(cuda_stream=7))
    for name in ("_raw_stream", "_device"):
        with monkeypatch.context() as m:
            m.setattr(ops, name, None)
            assert ops._stream() == 7


def test_product_never_imports_the_oracle():
    pkg = os.path.join(ROOT, "nano_qwen_b200")
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                src = open(os.path.join(dirpath, f)).read()
                assert not re.search(r"^\s*(from|import)\s+oracle\b", src, flags=re.M), f
