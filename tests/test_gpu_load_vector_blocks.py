"""The one-pass P1 load vector: blocks of 512 elements and their ends, shared and isolated
nodes, values that spread too far for a block's common scale, zeros, Inf and NaN, the
full mass table, and meshes whose blocks do not fit the stage -- against the oracle."""
import numpy as np
import pytest

import oracle as orc
from helpers import disjoint_tets
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _mesh(kind):
    if kind == "disjoint":  # 2048 nodes a block: the two-pass form
        return disjoint_tets(700)
    if kind == "isolated":  # nodes outside every element
        m = meshgen.kuhn_cube(5, jitter=0.2, seed=2, permute=True)
        conn = m.conn[(m.conn < 100).all(axis=1)]
        return m.xyz, np.ascontiguousarray(conn)
    m = meshgen.kuhn_cube(int(kind), jitter=0.2, seed=2, permute=True)
    return m.xyz, m.conn


def _run(xyz, conn, f, s, quad):
    import morganapublic_gb300 as mg
    mesh = mg.Mesh(xyz, conn, order=1)
    b = mg.MatrixBuilder(mesh)
    got = b.build_vector(field=f, elem_scale=s, quad=quad).cpu().numpy()
    again = b.build_vector(field=f, elem_scale=s, quad=quad).cpu().numpy()
    assert np.array_equal(got, again, equal_nan=True)  # bitwise reproducible
    return got, mesh


def _magnitude(xyz, conn, f, s, n):
    """Per node the sum of its entries' sizes, all products positive."""
    det = np.abs(meshgen.element_dets(xyz, conn))
    fa, sa = (np.ones(n) if f is None else np.abs(f)), (np.ones(len(conn)) if s is None else np.abs(s))
    y = (fa[conn].sum(1) * sa * det / 120.0)[:, None] + fa[conn] * (sa * det / 120.0)[:, None]
    out = np.zeros(n)
    np.add.at(out, conn.ravel(), y.ravel())
    return out


@pytest.mark.parametrize("kind", ["1", "2", "5", "11", "isolated", "disjoint"])
@pytest.mark.parametrize("quad", [1, 4, 64])
@pytest.mark.parametrize("decades", [0, 4, 30])
def test_blocks_match_oracle(kind, quad, decades):
    xyz, conn = _mesh(kind)
    rng = np.random.default_rng(7)
    f = rng.uniform(-1, 1, len(xyz)) * 10.0 ** rng.uniform(-decades, decades, len(xyz))
    s = rng.uniform(0.5, 1, len(conn)) * 10.0 ** rng.uniform(-decades, decades, len(conn))
    f[::7] = 0.0
    for ff, ss in ((f, s), (None, s), (f, None)):
        got, _ = _run(xyz, conn, ff, ss, quad)
        ref = orc.assemble_rhs(1, quad, xyz, conn, conn, len(xyz), field=ff, elem_scale=ss)
        # double-words: products and sums to ~2^-45 of the entries' sizes
        assert np.all(np.abs(got - ref) <= 1e-13 * _magnitude(xyz, conn, ff, ss, len(xyz)))


def test_special_values():
    xyz, conn = _mesh("11")
    rng = np.random.default_rng(3)
    f, s = rng.uniform(1, 2, len(xyz)), rng.uniform(1, 2, len(conn))
    ref = orc.assemble_rhs(1, 4, xyz, conn, conn, len(xyz), field=f, elem_scale=s)
    for where, bad in (("f", np.nan), ("f", np.inf), ("s", np.nan), ("s", -np.inf)):
        g, t = f.copy(), s.copy()
        if where == "f":
            g[700] = bad
            touched = (conn == 700).any(axis=1)
        else:
            t[4000] = bad
            touched = np.arange(len(conn)) == 4000
        hit = np.unique(conn[touched])
        got, _ = _run(xyz, conn, g, t, 4)
        assert np.isnan(got[hit]).all()
        rest = np.setdiff1d(np.arange(len(xyz)), hit)
        assert np.all(np.abs(got[rest] - ref[rest]) <= 1e-13 * np.abs(ref[rest]))
    for g, t in ((np.zeros_like(f), s), (f, np.zeros_like(s)), (np.full_like(f, 1e-310), s)):
        assert np.all(_run(xyz, conn, g, t, 4)[0] == 0.0)
