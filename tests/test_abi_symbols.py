"""The shared library loads without a GPU and exports every entry point the header declares."""

from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest

from alignquant_b200 import _lib

HEADER = Path(__file__).resolve().parents[1] / "include" / "alignquant_b200.h"


def declared_symbols() -> list[str]:
    text = HEADER.read_text()
    return re.findall(r"AQ_API\s+[\w\s\*]+?\b(aq_\w+)\s*\(", text)


def test_header_symbols_are_exported_and_bound():
    names = declared_symbols()
    assert len(names) >= 9 and len(set(names)) == len(names)
    lib = ctypes.CDLL(str(_lib.library_path()))
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"
    assert set(names) == set(_lib.SIGNATURES), "ctypes signatures and header declarations differ"


def test_pure_host_entry_points():
    lib = _lib.load()
    assert lib.aq_version() >= 100
    assert lib.aq_prepared_bytes(2, 3, 4, 2) == 2048 + 4 * 2048 + 2 * 4096
    assert lib.aq_prepared_bytes(2, 3, 4, 1) < 0 and "t4 + t8" in _lib.last_error()
    assert lib.aq_linear_workspace_bytes(0, 1, 1, 0, 0) < 0
    assert lib.aq_linear_workspace_bytes(64, 4, 4, 0, 4) == 0  # explicit splits: cluster kernel, no scratch


@pytest.mark.parametrize("m", [33, 129, 4096])
def test_workspace_of_the_largest_layer_suffices_for_smaller_ones(m):
    """One buffer serves every layer: the size does not fall as a layer gets wider or longer, whatever passes it is cut into."""
    size = _lib.load().aq_linear_workspace_bytes
    widths = [*range(1, 40), 79, 80, 204, 205, 408, 409, 420, 544, 819, 1024, 2500]
    lengths = [1, 2, 3, 31, 40, 79, 80, 81, 127, 160, 272, 333, 334, 335, 340, 342, 455, 456, 500, 511, 512]
    table = [[size(m, n_j, n_k, 0, 0) for n_k in lengths] for n_j in widths]
    if m > 128:  # at fewer rows some layers take the kernel without a workspace
        assert all(a <= b for row in table for a, b in zip(row, row[1:]))
        assert all(a <= b for upper, lower in zip(table, table[1:]) for a, b in zip(upper, lower))
    most = size(4096, 2500, 512, 0, 0)
    assert 0 <= min(map(min, table)) and max(map(max, table)) <= most
    assert f"{most // 1000000} {most // 1000 % 1000:03d} {most % 1000:03d} bytes" in HEADER.read_text()


@pytest.mark.parametrize("n_k", [513, 1365, 1366, 20000])
@pytest.mark.parametrize("m,schedule", [(33, 0), (128, 0), (129, 0), (4096, 0), (2, 3), (129, 3)])
def test_k_above_the_gemm_limit_is_refused_with_a_message(m, schedule, n_k):
    """Size and plan queries answer for any K, and the call says what its limit is (no launch, so no GPU)."""
    lib = _lib.load()
    assert lib.aq_linear_workspace_bytes(m, 4, n_k, schedule, 0) == 0
    kernel, splits, workers = (ctypes.c_int32() for _ in range(3))
    assert lib.aq_linear_plan(m, 4, n_k, schedule, 0, *(ctypes.addressof(v) for v in (kernel, splits, workers))) == 0
    assert kernel.value == 1 and splits.value >= 1
    at = 1 << 20  # never read
    assert lib.aq_linear(at, at, _lib.AQ_SCALE_TOKEN, m, at, 4, n_k, None, schedule, 0, _lib.AQ_F32, at, None, 0, None, None) == -1
    assert "K up to 32768" in _lib.last_error()


def test_options_are_validated_and_read_back():
    """Process-wide options: set, read back, reject values outside their range (no GPU involved)."""
    lib = _lib.load()
    defaults = {
        _lib.AQ_OPT_PEER_POLL_LIMIT: 1 << 22, _lib.AQ_OPT_GEMM_ROUNDING: 0, _lib.AQ_OPT_GEMM_TILE: 0,
        _lib.AQ_OPT_GEMM_SPLIT: 0, _lib.AQ_OPT_DECODE_KERNEL: 0, _lib.AQ_OPT_QUANT_FUSION_TILES: 2400,
    }
    for option, value in defaults.items():
        assert lib.aq_get_option(option) == value
    changes = {
        _lib.AQ_OPT_PEER_POLL_LIMIT: 4096, _lib.AQ_OPT_GEMM_ROUNDING: 1, _lib.AQ_OPT_GEMM_TILE: 4,
        _lib.AQ_OPT_GEMM_SPLIT: 3, _lib.AQ_OPT_DECODE_KERNEL: _lib.AQ_DECODE_KERNEL_STREAMK, _lib.AQ_OPT_QUANT_FUSION_TILES: 0,
    }
    try:
        for option, value in changes.items():
            assert lib.aq_set_option(option, value) == 0, _lib.last_error()
            assert lib.aq_get_option(option) == value
        for option, bad in ((_lib.AQ_OPT_PEER_POLL_LIMIT, 1), (_lib.AQ_OPT_GEMM_ROUNDING, 2), (_lib.AQ_OPT_GEMM_TILE, 3),
                            (_lib.AQ_OPT_GEMM_SPLIT, 9), (_lib.AQ_OPT_DECODE_KERNEL, 3), (_lib.AQ_OPT_QUANT_FUSION_TILES, -1), (99, 0)):
            assert lib.aq_set_option(option, bad) < 0
        assert lib.aq_get_option(99) < 0
    finally:
        for option, value in defaults.items():
            assert lib.aq_set_option(option, value) == 0

