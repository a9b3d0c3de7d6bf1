"""FP32 assembly where an element's scale factor (coefficient over determinant) is above the
floats: its diagonal entries are infinite, not NaN, and rows without such an element are
as accurate as ever."""
import numpy as np
import pytest

import oracle as orc
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,coeff", [(1.0, 1.0), (1e-2, 3e36), (1e-4, 1e36), (2e-6, 1e36)])
@pytest.mark.parametrize("n", [2, 3, 9])
def test_scale_factor_above_the_floats(n, size, coeff):
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=3, permute=True)
    xyz = m.xyz * size
    kappa = np.random.default_rng(n).uniform(0.5, 2.0, len(m.conn))
    far = m.xyz[m.conn].mean(axis=1)[:, 0] > 0.5
    kappa[far] *= coeff
    b = mg.MatrixBuilder(mg.Mesh(xyz, m.conn, order=1))
    _, rp, ci, ref = orc.full_operator("stiff_kappa", 1, 4, xyz, m.conn, coeff=kappa)
    got = b.assemble("stiff_kappa", coeff=kappa, quad=4, prec="f32").cpu().numpy()
    b.status()
    row = np.repeat(np.arange(b.ndof), np.diff(rp))
    diag = got[row == ci]
    assert not np.isnan(diag).any() and (diag > 0).all()
    near = np.setdiff1d(np.arange(b.ndof), np.unique(m.conn[far])) if coeff > 1 else np.arange(b.ndof)
    scale = np.zeros(b.ndof)
    np.maximum.at(scale, row, np.abs(ref))
    at = np.isin(row, near)
    assert len(near) and np.all(np.abs(got[at] - ref[at]) <= 2e-6 * scale[row[at]])
