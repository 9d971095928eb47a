"""Host check of the offsets the operand pass of the split-precision path
reads complex blocks with: the place of a part in a block of up to 2^31 - 1
elements, beyond what 32 bits hold."""
import ctypes as C

import pytest


@pytest.mark.parametrize("row,col", [(0, 0), (3, 5), (2 ** 30 - 1, 0), (2 ** 30, 0), (5, 2 ** 30),
                                     (2 ** 30, 2 ** 30 - 2), (2 ** 31 - 2, 0), (0, 2 ** 31 - 2)])
def test_parts_of_complex_elements(engine, row, col):
    f = engine.dll.xmgd_emu_part_at
    f.restype, f.argtypes = C.c_int64, [C.c_int32, C.c_int32, C.c_int]
    for half in (0, 1):
        assert f(row, col, half) == 2 * (row + col) + half
