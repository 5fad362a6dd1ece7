"""The shared memory that the input pass of a convolution asks for decides how many of its blocks an SM
holds: its even share of the grid, where that is below the eight that fit by their threads."""
import ctypes as C

import pytest

from shflbw_sparse_nn_b200 import _cabi
from shflbw_sparse_nn_b200.build import build_fault_inject_library

SMS, SM_KB, BLOCK_KB, SYSTEM_KB = 148, 228, 227, 1       # of a B200: shared memory of an SM, of a block, taken per block


@pytest.mark.parametrize("has_last_pass", [0, 1])
def test_blocks_per_sm(has_last_pass):
    lib = _cabi.load_library(build_fault_inject_library())
    lib.shflbw_debug_relayout_smem.argtypes, lib.shflbw_debug_relayout_smem.restype = [C.c_longlong, C.c_int], C.c_int
    for blocks in [1, 2, SMS - 1, SMS, 10 * SMS, 1 << 31] + [k * SMS + d for k in range(1, 9) for d in (-1, 0, 1)]:
        smem = lib.shflbw_debug_relayout_smem(blocks, has_last_pass)
        assert 16 << 10 <= smem <= BLOCK_KB << 10
        fit = min(8, (SM_KB << 10) // (smem + (SYSTEM_KB << 10)))
        share = -(-blocks // SMS)
        assert fit == (8 if share > 7 or (share == 1 and has_last_pass) else share)
