"""uns_cc_fvresidual after uns_cc_set_state: the state the caller hands in
brings ghost rows of its own, and a call gives every ghost row the boundary
closure's value (CCFVM/fvresidual.F90:27-100), whether it recomputes all faces
or, nothing but the conserved state having changed, the boundary faces alone."""
import numpy as np
import pytest

from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("flux", ["roe", "rusanov"])
def test_ghost_rows_after_set_state_are_those_of_a_full_call(precision, flux):
    m = mesh.CCMesh.airfoil(24, 10)
    p = abi.make_params(flux=flux, grad="gg", m_inf=0.6, aoa_deg=2.0, precision=precision)
    cfl = mesh.cfl_schedule(p, 1, 9, "cc")
    short, full = CCSolver(m, p), CCSolver(m, p)
    noc = m.ncells
    for s in (short, full):
        s.iterate(cfl[:8], first_iter=True)
        s.con2prim(); s.avg_c2v(); s.time_step(float(cfl[8])); s.save_old(); s.gradient()
        s.fvresidual()
        q = s.get_state()
        riemann = q[noc:].copy()
        q[:noc] *= 1.0 + 1e-3 * np.random.default_rng(3).random((noc, 1))
        q[noc:] = 7.0  # a caller that keeps the interior rows alone up to date
        s.set_state(q)
    full.set_precision(precision)  # every face again
    for s in (short, full):
        s.fvresidual()
    assert np.array_equal(short.get_state(), full.get_state())
    assert np.array_equal(short.get("res"), full.get("res"))
    far = m["fbc"][m["nfi"]:] == 2001
    assert far.any() and np.array_equal(short.get_state()[noc:][far], riemann[far])
    # and the stages after it, which nothing but the state's rows change
    for s in (short, full):
        s.rk_stage(1)
        s.fvresidual()
    assert np.array_equal(short.get_state(), full.get_state())
