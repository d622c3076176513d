"""LU-SGS sweep items with more neighbours than one pass of a warp takes (eight):
a disc whose centre node has 24 or 31 edges, numbered so that the centre comes
first (its backward item waits for all of them) and last (its forward item
does).  FP64: the oracle's operations in its order, so 1e-12 of the largest
value.  FP32 sweeps: the change dq against the FP64 form's.  A term is some
twenty FP32 operations of 2^-24 each on values of dq's own size, and a chain of
the disc's dozen levels adds up its items' errors: 24 x 20 x 2^-24 = 3e-5 of
the largest change."""
import numpy as np
import pytest

from oracle import OracleNC
from unsflow2d_gb300 import abi, mesh
from unsflow2d_gb300.solver import NCSolver

pytestmark = pytest.mark.gpu


def _disc(path, spokes, rings=5):
    """A disc in the geometry.inp layout: node 0 the centre, then the rings; the rim is farfield."""
    ang = 2 * np.pi * np.arange(spokes) / spokes
    rad = 0.3 * 1.5 ** np.arange(rings)
    x = np.concatenate([[0.0], *(r * np.cos(ang) for r in rad)])
    y = np.concatenate([[0.0], *(r * np.sin(ang) for r in rad)])
    node = lambda r, k: 1 + r * spokes + k % spokes  # noqa: E731
    tri = [(0, node(0, k), node(0, k + 1)) for k in range(spokes)]
    for r in range(rings - 1):
        for k in range(spokes):
            tri += [(node(r, k), node(r + 1, k), node(r + 1, k + 1)), (node(r, k), node(r + 1, k + 1), node(r, k + 1))]
    left = {(t[i], t[(i + 1) % 3]): c for c, t in enumerate(tri) for i in range(3)}  # directed edge -> cell to its left
    rim = [(node(rings - 1, k + 1), node(rings - 1, k)) for k in range(spokes)]
    with open(path, "w") as f:
        f.write(f"{len(x)} {len(tri)} {(len(left) + spokes) // 2}\n")
        for i in range(len(x)):
            f.write(f"{i + 1} {x[i]:.17g} {y[i]:.17g} {2001 if i >= node(rings - 1, 0) else 0}\n")
        for c, (a, b, d) in enumerate(tri):
            area = 0.5 * ((x[b] - x[a]) * (y[d] - y[a]) - (x[d] - x[a]) * (y[b] - y[a]))
            f.write(f"{c + 1} {(x[a] + x[b] + x[d]) / 3:.17g} {(y[a] + y[b] + y[d]) / 3:.17g} {area:.17g}\n")
        k = 0
        for (a, b), c in left.items():
            if a < b and (b, a) in left:
                k += 1
                f.write(f"{k} {a + 1} {b + 1} {c + 1} {left[b, a] + 1} {y[b] - y[a]:.17g} {x[a] - x[b]:.17g} 0\n")
        for a, b in rim:
            k += 1
            f.write(f"{k} {a + 1} {b + 1} 0 {left[b, a] + 1} {y[b] - y[a]:.17g} {x[a] - x[b]:.17g} 2001\n")


def _reversed(a):
    """The same mesh with its nodes numbered from the end."""
    n = int(a["nop"])
    out = dict(a)
    for k in ("px", "py", "cv"):
        out[k] = a[k][::-1].copy()
    for k in ("fp1", "fp2"):
        out[k] = (n - 1 - a[k]).astype(np.int32)
    for off, lists in (("v2v_off", ("v2v", "wx", "wy")), ("v2f_off", ("v2f",))):
        rows = np.concatenate([np.arange(a[off][i], a[off][i + 1]) for i in reversed(range(n))])
        out[off] = np.concatenate([[0], np.cumsum(np.diff(a[off])[::-1])]).astype(np.int32)
        for k in lists:
            out[k] = a[k][rows].copy()
    out["v2v"] = (n - 1 - out["v2v"]).astype(np.int32)
    return out


@pytest.mark.parametrize("last", [False, True], ids=["centre_first", "centre_last"])
@pytest.mark.parametrize("spokes", [24, 31])
def test_items_with_many_neighbours(tmp_path, spokes, last):
    _disc(tmp_path / "disc.inp", spokes)
    m = mesh.NCMesh.read(str(tmp_path / "disc.inp")).arrays
    if last:
        m = _reversed(m)
    centre = int(m["nop"]) - 1 if last else 0
    assert np.diff(m["v2f_off"])[centre] == spokes
    p = abi.make_params(flux="ausm", limiter="barth_corrected", time="lusgs", cfl_max=20.0, m_inf=0.4, aoa_deg=3.0)
    g, o, f = NCSolver(m, p), OracleNC(m, p), NCSolver(m, p)
    f.set_precision("mixed_sweep")
    rng = np.random.default_rng(8)
    q = g.get_state() * (1.0 + 0.01 * rng.standard_normal((int(m["nop"]), 4)))
    for s in (g, f):
        s.set_state(q)
    o.set("qc", q)
    for s in (g, o, f):
        s.save_old()
        s.lusgs(5.0)
    dq = g.get_state() - q
    assert np.max(np.abs(dq[centre])) > 0
    assert np.max(np.abs(g.get_state() - o.get_state())) <= 1e-12 * np.max(np.abs(o.get_state()))
    assert np.max(np.abs(f.get_state() - q - dq)) <= 3e-5 * np.max(np.abs(dq))
