"""The line of the launch chooser between two rows and one row per warp for long rows (pure host arithmetic)."""
import ctypes

import pytest

from macko_spmv_b200 import cabi


@pytest.mark.parametrize("rows,cols,row_length,lanes", [
    (5504, 11008, 8192, 16), (5504, 11008, 8208, 16), (5504, 11008, 12288, 16), (5504, 11008, 12304, 32),   # every warp holds one block of two rows
    (9472, 12000, 9000, 16), (9476, 12000, 9000, 32),                                                        # 4736 warps on 148 SMs: one block too many
    (5504, 16400, 9000, 32),                                                                                 # beyond 16384 columns chains stay short
])
def test_long_rows(rows, cols, row_length, lanes):
    lib = cabi.load()
    L, D = ctypes.c_int(), ctypes.c_int()
    cabi.check(lib, lib.macko_spmv_shape(rows, cols, rows * row_length, 148, ctypes.byref(L), ctypes.byref(D)))
    assert (L.value, D.value) == (lanes, 6)
