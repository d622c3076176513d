"""Where a sweep warp looks for its neighbours' records (host side, no GPU): in
its block's shared memory under (warp of the block, list index) where a warp of
the same block of four computes the neighbour, else in global memory.  A wrong
source would hand an item another item's record."""
import ctypes as C

import numpy as np
import pytest

from test_sweep_schedule import I32, _cc_graph, _nc_graph, _preds, _schedule
from unsflow2d_gb300 import abi, mesh


def _check(off, nbr, nwarps):
    woff, items, _ = _schedule(off, nbr, nwarps)
    lib = abi.host_lib()
    lib.uns_host_sweep_sources.argtypes = [C.c_int, I32, I32, C.c_int, I32, I32]
    off, nbr = np.ascontiguousarray(off, dtype=np.int32), np.ascontiguousarray(nbr, dtype=np.int32)
    src, nsrc = np.full(len(nbr) + 1, -7, dtype=np.int32), np.zeros(1, dtype=np.int32)
    p = lambda a: a.ctypes.data_as(I32)  # noqa: E731
    assert lib.uns_host_sweep_sources(len(off) - 1, p(off), p(nbr), nwarps, p(src), p(nsrc)) == 0
    place = {}  # item code -> (warp, list index)
    for w in range(nwarps):
        for k in range(woff[w], woff[w + 1]):
            place[int(items[k])] = (w, k - int(woff[w]))
    want = []
    for w in range(nwarps):
        for k in range(woff[w], woff[w + 1]):
            code = int(items[k])
            for q in _preds(off, nbr, code)[code & 1:]:  # a backward item's own forward value has no source
                v, idx = place[q]
                want.append((v % 4) << 28 | idx if v // 4 == w // 4 else -1)
    assert int(nsrc[0]) == len(want) and np.array_equal(src[:len(want)], want)
    return np.array(want)


@pytest.mark.parametrize("nwarps", [1, 4, 6, 64, 608])
def test_nc_sources(nwarps):
    want = _check(*_nc_graph(mesh.NCMesh.airfoil(32, 16)), nwarps)
    assert np.any(want >= 0) and (nwarps <= 4 or np.any(want < 0))


@pytest.mark.parametrize("nwarps", [5, 96])
def test_cc_sources(nwarps):
    _check(*_cc_graph(mesh.CCMesh.airfoil(32, 16)), nwarps)


@pytest.mark.parametrize("seed", range(6))
def test_sources_on_random_graphs(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 400))
    off = np.concatenate([[0], np.cumsum(rng.integers(0, 9, n))]).astype(np.int32)
    nbr = rng.integers(-3, n + 3, int(off[-1])).astype(np.int32)
    _check(off, nbr, int(rng.integers(1, 40)))
