"""The FP32 product with infinite entries, sums that overflow, and NaN: the streamed kernel
(P2, 32-bit columns) and the others (P1) give the values of IEEE sums, and the
rows beside them stay as they are."""
import numpy as np
import pytest

from helpers import star_mesh
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _builder(kind):
    import morganapublic_gb300 as mg
    if kind == "star":
        xyz, conn = star_mesh(9000)
        return mg.MatrixBuilder(mg.Mesh(xyz, conn, order=2))
    m = meshgen.kuhn_cube(18 if kind == "p2" else 9, jitter=0.1, seed=4, permute=True)
    return mg.MatrixBuilder(mg.Mesh(m.xyz, m.conn, order=2 if kind == "p2" else 1))


@pytest.mark.parametrize("kind", ["p2", "star", "p1"])
def test_nonfinite_rows(kind):
    import torch
    b = _builder(kind)
    rp, ci = b.pattern()
    if kind != "p1":
        row = np.repeat(np.arange(b.ndof), np.diff(rp))
        assert np.max(np.abs(ci - row)) > 32767 and b.nnz > 16 * b.ndof  # the streamed kernel's rule
    rng = np.random.default_rng(1)
    vals = rng.uniform(-1.0, 1.0, b.nnz).astype(np.float32)
    plain = b.apply(torch.from_numpy(vals).cuda(), torch.ones(b.ndof, device="cuda")).cpu().numpy()
    inf, want, at = np.float32(np.inf), {}, 1
    longest = int(np.argmax(np.diff(rp)))

    def put(row, where, value, result):
        k = rp[row] + where if where >= 0 else rp[row + 1] + where
        vals[k] = value
        want[row] = result

    for value in (inf, -inf, np.float32(np.nan)):
        for where in (0, 1, -1):
            put(at, where, value, value)
            at += 16 + at % 3
    put(at, 0, inf, np.nan)   # opposite infinities
    put(at, 1, -inf, np.nan)
    at += 7
    for sign in (1.0, -1.0):  # finite entries whose sum is above FP32's range
        vals[rp[at]:rp[at + 1]] = np.float32(sign * 1e38)
        want[at] = sign * inf
        at += 21
    put(longest, -2, -inf, -inf)
    assert at < b.ndof and longest not in list(want)[:-1]
    y = b.apply(torch.from_numpy(vals).cuda(), torch.ones(b.ndof, device="cuda")).cpu().numpy()
    for row, w in want.items():
        assert np.array_equal(y[row], np.float32(w), equal_nan=True), (row, w, y[row])
    rest = np.setdiff1d(np.arange(b.ndof), list(want))
    assert np.array_equal(y[rest], plain[rest])
