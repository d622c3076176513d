"""Graph-replayed iterations vs the oracle on meshes either side of the sizes
where the FP64 launches change (products on the FP64 unit or on the integer
pipe, 128 or 256 threads: at 2 x 256 elements per SM), on sizes that leave
ragged blocks, and on the smallest mesh; the LU-SGS ones are long enough for a
sweep block's shared-memory boxes to be used many times over.

Criterion: the bound that the 60-iteration histories keep to elsewhere, 1e-10
of the largest state and 1e-9 in the logarithm of the norm.  Every operation is
rounded as the oracle's, so only pow may differ in its last bits.
"""
import numpy as np
import pytest

from oracle import OracleCC, OracleNC
from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import CCSolver, NCSolver

pytestmark = pytest.mark.gpu

RK3 = dict(flux="roe", grad="gg", m_inf=0.6, aoa_deg=2.0)
RAMP = dict(time="lusgs", cfl_max=5.0, cfl_type="ramp", cfl_min=0.5, cfl_ramp_steps=10)
NC_SGS = dict(flux="ausm", limiter="barth_corrected", time="lusgs", cfl_max=50.0, m_inf=0.8, aoa_deg=1.25)


@pytest.mark.parametrize("kind,ni,nj,case", [
    ("cc", 8, 3, RK3),
    ("cc", 241, 161, RK3),  # 77 602 cells: below 77 824
    ("cc", 244, 160, RK3),  # 78 080 cells: above
    ("cc", 244, 160, dict(RK3, **RAMP)),
    ("cc", 121, 67, dict(flux="roe", grad="ggfc", flow="laminar", iwall=0, rey=500.0, m_inf=0.5)),
    ("nc", 480, 160, NC_SGS),  # 77 280 nodes
    ("nc", 483, 161, dict(flux="vanleer", limiter="vkn", time="rk3", cfl_max=0.9, m_inf=0.6, aoa_deg=2.89)),  # 78 246
], ids=["smallest", "below", "above", "lusgs", "laminar", "nc_lusgs", "nc_rk3"])
def test_iterations_either_side_of_the_launch_rules(kind, ni, nj, case):
    M, S, Orc = (mesh.CCMesh, CCSolver, OracleCC) if kind == "cc" else (mesh.NCMesh, NCSolver, OracleNC)
    m, p = M.airfoil(ni, nj), abi.make_params(**case)
    g, o = S(m, p), Orc(m, p)
    cfl = mesh.cfl_schedule(p, 1, 3, kind)
    f = g.iterate(cfl, first_iter=True)
    norms = [o.iteration(c) for c in cfl]
    if kind == "nc":
        f, norms = f[0], [n[0] for n in norms]
    assert np.max(np.abs(np.log10(f / np.array(norms)))) < 1e-9
    assert np.max(np.abs(g.get_state() - o.get_state())) <= 1e-10 * np.max(np.abs(o.get_state()))
