"""The streamed FP32 SpMV (32-bit columns, long rows): rows around a warp's 16, around
the shared-memory window and its batches, against FP64 sums of the same entries."""
import numpy as np
import pytest

from helpers import star_mesh
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _check(b, seed):
    import torch
    rp, ci = b.pattern()
    rng = np.random.default_rng(seed)
    vals = rng.uniform(-1.0, 1.0, b.nnz).astype(np.float32)
    x = rng.uniform(-1.0, 1.0, b.ndof).astype(np.float32)
    y = b.apply(torch.from_numpy(vals).cuda(), torch.from_numpy(x).cuda()).cpu().numpy()
    p = vals.astype(np.float64) * x[ci].astype(np.float64)
    ref = np.add.reduceat(p, rp[:-1])
    mag = np.add.reduceat(np.abs(p), rp[:-1])
    # a product is rounded once (2^-24 of its size); their compensated sum once at the end
    assert np.all(np.abs(y - ref) <= 2.0 ** -23 * mag)


@pytest.mark.parametrize("n", [17, 18, 19])
def test_streamed_spmv_p2(n):
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.1, seed=4, permute=True)
    b = mg.MatrixBuilder(mg.Mesh(m.xyz, m.conn, order=2))
    rp, ci = b.pattern()
    row = np.repeat(np.arange(b.ndof), np.diff(rp))
    assert np.max(np.abs(ci - row)) > 32767 and b.nnz > 16 * b.ndof  # the streamed kernel's rule
    _check(b, n)


def test_streamed_spmv_long_row():
    """A row of 45,000 entries: many windows."""
    import morganapublic_gb300 as mg
    xyz, conn = star_mesh(9000)
    b = mg.MatrixBuilder(mg.Mesh(xyz, conn, order=2))
    rp, ci = b.pattern()
    assert np.max(np.diff(rp)) > 40000 and np.max(ci) > 40000 and b.nnz > 16 * b.ndof
    _check(b, 3)
