"""uns_cc_lusgs on packed cases, which have no sweep schedule: an error status,
and a handle that goes on as if the call had not been made."""
import numpy as np
import pytest

from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCPacked

pytestmark = pytest.mark.gpu


def test_lusgs_is_refused_and_the_handle_goes_on():
    meshes = [mesh.CCMesh.airfoil(16, 8), mesh.CCMesh.airfoil(17, 9)]
    params = [abi.make_params(m_inf=0.5), abi.make_params(m_inf=0.6)]
    cfl = np.stack([mesh.cfl_schedule(p, 1, 6, "cc") for p in params])
    a, b = CCPacked(meshes, params), CCPacked(meshes, params)
    a.iterate(cfl[:, :3], first_iter=True)
    b.iterate(cfl[:, :3], first_iter=True)
    assert a._lib.uns_cc_lusgs(a._h) == abi.UNS_ERR_ARG
    a.iterate(cfl[:, 3:], first_iter=False)
    b.iterate(cfl[:, 3:], first_iter=False)
    for i in range(2):
        assert np.array_equal(a.get_state(i), b.get_state(i))
