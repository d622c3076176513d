"""How a block of threads finds the packed case it works on (host side, no GPU).

A case's cells are padded to a multiple of 256 and the padding belongs to no
case (instance -1), so a block narrower than that can be padding from its
first cell on.  At every block width the kernels use, the cell by which a
block looks up its case must be a real one, of the case that holds the block."""
import ctypes as C

import numpy as np
import pytest

from unsflow2d_gb300 import abi

I32 = C.POINTER(C.c_int32)


@pytest.mark.parametrize("threads", [32, 64, 128, 256])
def test_every_block_finds_a_real_cell_of_its_case(threads):
    rng = np.random.default_rng(4)
    cells = np.concatenate([[576, 1, 255, 256, 257, 512, 513, 32, 33], rng.integers(1, 5000, 30)]).astype(np.int32)
    n = len(cells)
    lib = abi.host_lib()
    lib.uns_host_packed_layout.argtypes = [C.c_int, I32, C.c_int, I32, I32]
    first = np.zeros(n + 1, dtype=np.int32)
    block_cell = np.full(int(np.sum(cells + 256)) // threads + 1, -1, dtype=np.int32)
    p = lambda a: a.ctypes.data_as(I32)  # noqa: E731
    assert lib.uns_host_packed_layout(n, p(cells), threads, p(first), p(block_cell)) == 0
    inst = np.full(int(first[-1]), -1)
    for i in range(n):
        assert first[i] % 256 == 0 and first[i + 1] >= first[i] + cells[i]
        inst[first[i]:first[i] + cells[i]] = i
    owner = np.repeat(np.arange(n), np.diff(first))
    blocks = int(first[-1]) // threads
    starts = np.arange(blocks) * threads
    if threads < 256:
        assert np.any(inst[starts] == -1)  # some blocks do begin in padding
    assert np.array_equal(inst[block_cell[:blocks]], owner[starts])
