"""B from face areas and per-card tables, and the saddle gather with four entries
per thread, against the oracle: one element's surface, entries with more and fewer
than four sources, sizes around the kernels' blocks, every test basis."""
import numpy as np
import pytest

import oracle as orc
from helpers import row_scaled_err
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu

# an entry sums at most about 10 equal-sign terms, each area2 (10 roundings of 2^-53)
# times a table entry (12), on both sides: below 2 x 32 x 2^-53 of its row's largest
TOL = 64 * 2.0**-53


@pytest.mark.parametrize("n,order,test_order,quad", [(1, 1, 1, 1), (1, 2, 2, 6), (2, 1, 0, 4), (3, 2, 0, 6), (5, 1, 2, 6),
                                                     (6, 2, 1, 4), (9, 1, 1, 3), (13, 1, 1, 6)])
def test_boundary_values(n, order, test_order, quad):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=n, permute=True)
    mesh = mg.Mesh(m.xyz, m.conn, order=order)
    b = mg.MatrixBuilder(mesh)
    tris = None
    if test_order == 0:
        fe, fl = orc.boundary_faces(m.conn)
        tris = m.conn[fe[:, None], orc.FACE_PTS[fl]]
    lg = mg.LagrangeBuilder(b, tris=tris, test_order=test_order)
    K = b.assemble("stiff_const")
    B = lg.assemble(quad=quad)
    S = lg.saddle(K, B)
    dofs = mesh.elem_dofs()
    _, rp, ci, ref, _, _ = orc.lagrange(order, quad, m.xyz, m.conn, dofs, b.ndof, tris=tris, test_order=test_order)
    (brp, bci), (srp, sci) = lg.pattern()
    assert np.array_equal(brp, rp) and np.array_equal(bci, ci)
    assert row_scaled_err(rp, ref, B.cpu().numpy()) <= TOL
    krp, kci = b.pattern()
    osrp, osci, sref = orc.saddle(krp, kci, K.cpu().numpy(), rp, ci, B.cpu().numpy(), b.ndof)
    assert np.array_equal(srp, osrp) and np.array_equal(sci, osci)
    assert np.array_equal(S.cpu().numpy(), sref)  # copies
    # the areas of the first card stay in use while the second card's gather runs
    other = lg.assemble(quad=1)
    assert torch.equal(lg.assemble(quad=quad), B) and other.shape == B.shape
