"""The load vector at the ends of FP64: field, element scale and mesh multiplied by
powers of two, which multiply the result exactly -- against the oracle's result on the
unscaled inputs, times the same power (Inf above the range, rounded below it)."""
import numpy as np
import pytest

import oracle as orc
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,quad", [(1, 4), (5, 4), (5, 1), (5, 64)])
@pytest.mark.parametrize("a,b,c", [
    (-1016, -1016, (0, 0, 0)),   # far below the range: zero
    (-1020, -1021, (0, 0, 0)),
    (-1020, -1021, (-2, -2, -2)),  # total powers of -2047, -2050 and below
    (-1020, -1021, (-3, -3, -3)),
    (-1021, -1021, (-20, -21, -20)),
    (-1000, -1000, (30, 30, 30)),
    (1016, 1016, (0, 0, 0)),     # far above: Inf
    (1021, 1020, (0, 0, 0)),
    (1021, 1000, (40, 41, 41)),
    (1021, 1021, (3, 3, 3)),
    (1022, 1022, (42, 42, 42)),
    (1000, -1021, (40, 40, 40)),
    (-1021, 1000, (-30, -30, -30)),
    (-1016, 1016, (0, 0, 0)),    # the ends cancel
    (1016, -1016, (-10, 5, 3)),
    (-530, -530, (0, 0, 0)),     # around the smallest doubles
    (520, 510, (0, 0, 0)),       # around the largest
    (3, -4, (42, 42, 42)),       # determinants of 2^126, 2^127
    (3, -4, (43, 42, 42)),
    (-500, -560, (42, 42, 42)),
])
def test_powers_of_two(n, quad, a, b, c):
    import morganapublic_gb300 as mg
    # coordinates of few bits: determinants and products exact at every power
    m = meshgen.kuhn_cube(n, jitter=0.0, permute=True, seed=3)
    xyz = np.round(m.xyz * n)
    rng = np.random.default_rng(5)
    f, s = rng.uniform(1, 2, len(xyz)), rng.uniform(1, 2, len(m.conn))
    ref = orc.assemble_rhs(1, quad, xyz, m.conn, m.conn, len(xyz), field=f, elem_scale=s)
    moved = np.ldexp(xyz, np.array(c))
    bld = mg.MatrixBuilder(mg.Mesh(moved, m.conn, order=1))
    got = bld.build_vector(field=np.ldexp(f, a), elem_scale=np.ldexp(s, b), quad=quad).cpu().numpy()
    k = a + b + sum(c)
    with np.errstate(over="ignore", under="ignore"):
        want = np.ldexp(ref, k)
    tiny = 2.0 ** -1074
    assert np.array_equal(np.isinf(got), np.isinf(want)) and not np.isnan(got).any()
    fin = np.isfinite(want)
    # all inputs positive: 1e-13 of the value, and below the normal range half a unit per
    # partial sum (a node lies in two blocks at most here)
    assert np.all(np.abs(got[fin] - want[fin]) <= 1e-13 * want[fin] + 2 * tiny)
