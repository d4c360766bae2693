"""Rows that the attention backward's row products take, over the whole range that the entry point accepts."""
import ctypes

import pytest

from mist_b200.ops import native

ROWS, GROUPS = 4, 16         # rows of a thread group, groups of a block (attn_delta_kernel)


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 2 ** 28, 2 ** 30 - 1, 2 ** 30 + 1, 2 ** 31 - 1])
def test_every_row_has_its_group(rows):
    if not native.kernels_path().exists():
        pytest.skip("the kernels library is not built")
    lib = ctypes.CDLL(str(native.kernels_path()))
    first = lib.mb_attn_delta_first_row
    first.argtypes, first.restype = [ctypes.c_uint, ctypes.c_uint], ctypes.c_uint
    blocks = -(-rows // (ROWS * GROUPS))
    for block in {0, blocks // 3, blocks // 2, blocks - 1}:
        for group in (0, 1, GROUPS - 1):
            for thread in (16 * group, 16 * group + 15):
                assert first(block, thread) == (block * GROUPS + group) * ROWS
    assert first(blocks - 1, 255) + ROWS >= rows
