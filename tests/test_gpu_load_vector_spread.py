"""Load vectors of fields whose values spread by more than 2^70 within the blocks (sharp
bumps, far values, subnormal ones, zeros), beside element scales that do: against sums of
the oracle's entries in extended precision, by each node's own size."""
import numpy as np
import pytest

import oracle as orc
from helpers import disjoint_tets
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _reference(xyz, conn, f, s, quad):
    """Per node the sum and the sum of sizes of its entries, from element-wise exact powers of two."""
    n, ld = len(xyz), np.longdouble
    det = np.abs(meshgen.element_dets(xyz, conn)).astype(ld)
    fe = (np.ones((len(conn), 4)) if f is None else f[conn]).astype(ld)
    se = (np.ones(len(conn)) if s is None else s).astype(ld)
    one = np.arange(4, dtype=np.int32)[None]
    M = np.array([orc.assemble_rhs(1, quad, np.eye(4, 3, k=-1), one, one, 4, field=np.eye(4)[k])
                  for k in range(4)]).astype(ld)
    y = np.einsum("lk,ek->el", M.T, fe) * (se * det)[:, None]
    a = np.einsum("lk,ek->el", np.abs(M.T), np.abs(fe)) * (np.abs(se) * det)[:, None]
    out, mag = np.zeros(n, ld), np.zeros(n, ld)
    np.add.at(out, conn.ravel(), y.ravel())
    np.add.at(mag, conn.ravel(), a.ravel())
    return out, mag


@pytest.mark.parametrize("quad", [1, 4, 64])
@pytest.mark.parametrize("field", ["bump", "far", "tiny", "subnormal", "high", "none"])
@pytest.mark.parametrize("n", [1, 5, 12, 20])
def test_spread(n, field, quad):
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2 if n > 1 else 0.0, seed=2, permute=True)
    rng = np.random.default_rng(n)
    N, E = len(m.xyz), len(m.conn)
    f, s = rng.uniform(-2, 2, N), rng.uniform(0.5, 2, E)
    if field == "bump":
        f = np.exp(-((m.xyz - 0.45) ** 2).sum(1) / (2 * 0.02 ** 2))
    elif field == "far":
        f[::13] = 1e-30
    elif field == "tiny":  # the smallest normal numbers and below beside others
        f *= np.where(rng.random(N) < 0.3, 3e-308, 1e-290)
        s *= 1e100
    elif field == "subnormal":
        f = np.where(rng.random(N) < 0.5, rng.integers(1, 1 << 40, N) * 2.0 ** -1074, 4e-308 * f)
        s *= 1e150
    elif field == "high":
        f *= 10.0 ** rng.uniform(200, 306, N)
        s *= 10.0 ** rng.uniform(-180, -100, E)
    elif field == "none":
        f, s = None, s * 10.0 ** rng.uniform(-140, 140, E)
    b = mg.MatrixBuilder(mg.Mesh(m.xyz, m.conn, order=1))
    got = b.build_vector(field=f, elem_scale=s, quad=quad).cpu().numpy()
    assert np.array_equal(got, b.build_vector(field=f, elem_scale=s, quad=quad).cpu().numpy())
    fs = f if f is None else np.where(np.abs(f) < 2.0 ** -1022, 0.0, f)
    dead = np.zeros(E, bool) if f is None else (fs[m.conn] == 0).all(axis=1)  # all subnormal: zero by rule
    ref, mag = _reference(m.xyz, m.conn, f, np.where(dead, 0.0, s), quad)
    # an element's vector to 2^-45 of its sizes, then FP64 sums; below the normal range every
    # entry is rounded to the doubles' spacing there
    entries = np.bincount(m.conn.ravel(), minlength=N)
    assert np.all(np.abs(got - ref) <= 1e-13 * mag + entries * np.longdouble(2) ** -1075)


@pytest.mark.parametrize("quad", [1, 4, 64])
@pytest.mark.parametrize("n", [5, 20])
@pytest.mark.parametrize("size", [1e-9, 1e9])
def test_spread_with_small_and_large_determinants(n, size, quad):
    # (size 1e-9, and an offset that keeps the coordinates near one: determinants of 2^-103)
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=2, permute=True)
    xyz = m.xyz * size + 1.0
    rng = np.random.default_rng(n)
    f, s = rng.uniform(-2, 2, len(xyz)), rng.uniform(0.5, 2, len(m.conn))
    f[::13] = 1e-30
    got = mg.MatrixBuilder(mg.Mesh(xyz, m.conn, order=1)).build_vector(field=f, elem_scale=s, quad=quad).cpu().numpy()
    ref, mag = _reference(xyz, m.conn, f, s, quad)
    assert np.all(np.abs(got - ref) <= 1e-13 * mag)
