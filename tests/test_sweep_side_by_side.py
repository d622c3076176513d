"""LU-SGS sweeps of several handles at once: the sweep of a mesh whose
dependency levels are narrow takes a part of the GPU's blocks (host side), and
handles batched in one graph evolve as they do alone, where their sweeps fit
beside each other and where they share the SMs."""

import numpy as np
import pytest

from test_sweep_schedule import _nc_graph, _schedule
from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCBatch, CCSolver

NSM = 152


@pytest.mark.parametrize("ni,nj,parts", [(64, 32, 3), (320, 160, 3), (512, 256, 2), (1024, 512, 1)])
def test_narrow_graphs_leave_blocks_to_other_sweeps(ni, nj, parts):
    off, nbr = _nc_graph_fast(mesh.NCMesh.airfoil(ni, nj))
    woff, items, lev = _schedule(off, nbr, 4 * NSM)
    used = np.flatnonzero(np.diff(woff)) // 4
    assert used.max() + 1 <= NSM // parts  # lists fill blocks from the first on
    # the other lists still hold two warps per item of an average level
    width = 2 * (len(off) - 1) / int(lev.sum())
    assert parts == 1 or 4 * (NSM // parts) >= 2 * width


def _nc_graph_fast(m):
    a = m.arrays
    off, e = a["v2f_off"], a["v2f"]
    own = np.repeat(np.arange(a["nop"]), np.diff(off))
    return off, np.where(a["fp2"][e] == own, a["fp1"][e], a["fp2"][e])


def test_graph_helper_agrees():
    m = mesh.NCMesh.airfoil(16, 8)
    assert all(np.array_equal(x, y) for x, y in zip(_nc_graph(m), _nc_graph_fast(m)))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed_sweep"])
@pytest.mark.parametrize("sizes", [[(24, 12), (30, 14)], [(128, 64), (96, 48), (128, 64), (120, 60)]],
                         ids=["beside", "sharing"])
def test_batched_sweeps_equal_handles_alone(sizes, precision):
    p = abi.make_params(flux="roe", grad="gg", m_inf=0.6, aoa_deg=2.0, time="lusgs", cfl_max=5.0, cfl_type="ramp",
                        cfl_min=0.5, cfl_ramp_steps=10, precision=precision)
    meshes = [mesh.CCMesh.airfoil(ni, nj) for ni, nj in sizes]
    batched, alone = [CCSolver(m, p) for m in meshes], [CCSolver(m, p) for m in meshes]
    cfl = mesh.cfl_schedule(p, 1, 12, "cc")
    b = CCBatch(batched)
    hist, done = b.iterate(np.tile(cfl, (len(meshes), 1)), first_iter=True)
    for i, s in enumerate(alone):
        h = s.iterate(cfl, first_iter=True)
        assert done[i] == 12 and np.array_equal(hist[i], h)
        assert np.array_equal(batched[i].get_state(), s.get_state())
    # a batched handle on its own afterwards
    more = mesh.cfl_schedule(p, 13, 3, "cc")
    batched[0].iterate(more, first_iter=False)
    alone[0].iterate(more, first_iter=False)
    assert np.array_equal(batched[0].get_state(), alone[0].get_state())
    b.close()
