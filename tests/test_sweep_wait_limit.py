"""The sweeps' wait bounds (host side, no GPU): whatever limit a caller sets, a
wait between the warps of a block is allowed at least as long as the wait for
another block's record, up to the largest value."""
import ctypes as C

import pytest

from unsflow2d_gb300 import abi

MAX = (1 << 63) - 1


@pytest.mark.parametrize("cycles", [1, 1000, 4_000_000_000, 1 << 40, (MAX - 100_000_000) // 4, (MAX - 100_000_000) // 4 + 1,
                                    MAX // 4, MAX // 2, MAX - 1, MAX])
def test_waits_inside_a_block_outlast_the_limit(cycles):
    lib = abi.host_lib()
    lib.uns_host_ring_wait_limit.argtypes, lib.uns_host_ring_wait_limit.restype = [C.c_int64], C.c_int64
    assert lib.uns_host_ring_wait_limit(cycles) >= min(MAX, 4 * cycles)
