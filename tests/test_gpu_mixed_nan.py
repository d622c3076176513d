"""A non-finite cell in the mixed form: FP32 arithmetic gives NaNs of one sign,
and the limiter range (a minimum and maximum over encoded keys, in which a
NaN's sign counts) must not depend on the signs that flux differences flip on
the way.  After a failed step, the limiter of the finite cells is the one that
the same state gives with its NaNs in the sign that FP32 arithmetic has."""
import numpy as np
import pytest

from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grad", ["gg", "lsqr"])
@pytest.mark.parametrize("by_routines", [False, True])
def test_limiter_range_beside_non_finite_cells(grad, by_routines):
    m = mesh.CCMesh.airfoil(30, 14)
    p = abi.make_params(flux="roe", grad=grad, m_inf=0.7, aoa_deg=2.0, precision="mixed")
    a, b = CCSolver(m, p), CCSolver(m, p)
    for s in (a, b):
        s.iterate(np.full(20, 0.8), first_iter=True)
        q = s.get_state()
        q[100:103] = np.nan
        s.set_state(q)
        with pytest.raises(abi.UnsError):
            if by_routines:
                s.iteration(0.8)
            else:
                s.iterate(np.full(2, 0.8), first_iter=False)
    q = b.get_state()
    bad = np.isnan(q)
    assert bad.any() and not bad.all()
    q[bad] = np.nan  # one sign
    b.set_state(q)
    phi = []
    for s in (a, b):
        s.set("phi", np.ones((s.noc, 4)))
        s.con2prim(); s.avg_c2v(); s.time_step(0.8); s.save_old(); s.gradient()
        phi.append(s.get("phi"))
    assert np.any(phi[1] < 1.0)
    assert np.array_equal(phi[0], phi[1], equal_nan=True)
