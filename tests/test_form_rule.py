"""The rule that picks the kernel of a composed-format product, asked through the library's query (nothing is
launched): widths, sizes of B and numbers of slots on both sides of every line."""
import ctypes

import numpy as np
import pytest

from liteform_ae_b200 import _cabi

GROUPS, SLOTS, RING, REGISTERS = ("spmm_hyb_groups_kernel", "spmm_hyb_ring_rows_kernel", "spmm_hyb_ring_kernel",
                                  "spmm_hyb_kernel")


def _name(dtype, N, cols, slots, ldb=None, ldc=None, parts=1):
    a = _cabi.LfHyb()
    off = np.array([0, slots], dtype=np.int64)
    a.num_rows, a.num_cols, a.num_parts, a.num_buckets = 1 << 20, cols, parts, 1
    a.slot_off = off.ctypes.data
    lib, ldb, ldc = _cabi.load(), ldb or N, ldc or N
    if dtype == "bf16":
        return lib.lf_spmm_hyb_bf16_kernel_name(ctypes.byref(a), ldb, ldc, N).decode()
    return lib.lf_spmm_hyb_f32_kernel_name(ctypes.byref(a), 0x1000, ldb, 0x2000, ldc, N).decode()


MANY, FEW = 1 << 24, (1 << 20) - 1


@pytest.mark.parametrize("N", [136, 144, 160, 192, 208, 240, 248, 392, 448, 504])
@pytest.mark.parametrize("cols", [1 << 19, 1 << 20, 1 << 22])
def test_bf16_rows_with_a_short_even_piece_keep_the_ring_per_warp(N, cols):
    assert _name("bf16", N, cols, MANY) == RING


@pytest.mark.parametrize("N", [256, 264, 320, 384, 512, 640, 768])
def test_bf16_rows_of_full_or_odd_pieces(N):
    assert _name("bf16", N, 1 << 19, MANY) == SLOTS
    assert _name("bf16", N, (1 << 19) - 1, MANY) == RING
    assert _name("bf16", N, 1 << 20, FEW) == RING


@pytest.mark.parametrize("dtype,N,cols,slots,name", [
    ("f32", 32, 851_968, MANY, GROUPS), ("f32", 32, 851_969, MANY, SLOTS), ("f32", 32, 1 << 22, FEW, GROUPS if 4 * 32 * FEW <= 104 << 20 else REGISTERS),
    ("f32", 64, 327_680, MANY, GROUPS), ("f32", 64, 327_681, MANY, SLOTS), ("f32", 64, 327_681, FEW, REGISTERS),
    ("f32", 68, 100_000, MANY, RING), ("f32", 128, 100_000, MANY, RING), ("f32", 68, 100_000, FEW, GROUPS), ("f32", 128, 100_000, FEW, GROUPS),
    ("f32", 132, 100_000, MANY, GROUPS), ("f32", 256, 100_000, MANY, RING), ("f32", 256, 80_000, MANY, GROUPS),
    ("bf16", 64, 851_968, MANY, GROUPS), ("bf16", 72, 100_000, MANY, SLOTS), ("bf16", 128, 100_000, FEW, GROUPS),
    ("bf16", 136, 1000, FEW, RING), ("f32", 47, 1000, MANY, REGISTERS)])
def test_lines(dtype, N, cols, slots, name):
    assert _name(dtype, N, cols, slots) == name


def test_float32_rows_that_fill_a_warp_go_by_groups_without_partitions_only():
    assert _name("f32", 128, 100_000, FEW, parts=4) == RING
    assert _name("f32", 64, 100_000, FEW, parts=4) == _name("f32", 160, 100_000, FEW, parts=4) == GROUPS


def test_pitches_beyond_32_bits_keep_the_registers():
    assert _name("f32", 32, 1000, MANY, ldb=1 << 30) == REGISTERS
    assert _name("f32", 64, 1000, MANY, ldc=1 << 30) == SLOTS
