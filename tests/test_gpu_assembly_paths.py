"""The P1 assembly's rules for its inputs: the split of the node coordinates (on
grids, or each remainder rounded, for meshes with very thin elements or large
offsets), coefficient arrays off the 16-byte grid or of odd length, and block
ends -- against the oracle."""
import numpy as np
import pytest

import oracle as orc
from helpers import row_scaled_err
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu

F64_TOL = 1e-12
F32_TOL = 2e-6


def _thin(m):
    """One layer of cells squeezed to 1e-7 of the cube: no grid split."""
    x = m.xyz.copy()
    first = np.isclose(x[:, 2], 1.0 / m.n)
    x[first, 2] = 1e-7
    return x


def _offset(m):
    """The cube moved far from the origin: cells of 2^-21 of the coordinates."""
    return m.xyz + np.array([3.0e5, -2.0e5, 1.0e5])


def _shifted(m):
    """Coordinates of both signs: the grid split with negative parts."""
    return 2.0 * m.xyz - np.array([1.0, 0.7, 0.3])


@pytest.mark.parametrize("move,drop,lead", [
    (None, 0, 0), (None, 1, 0), (None, 0, 1), (None, 1, 1),  # odd element counts, coefficient 8 bytes off
    (_shifted, 1, 1), (_offset, 0, 0), (_thin, 0, 0),
])
@pytest.mark.parametrize("n,op", [(2, "stiff_kappa"), (5, "stiff_kappa"), (5, "mass_coeff"), (11, "stiff_kappa")])
def test_assembly_paths_match_oracle(move, drop, lead, n, op):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.0 if move is _thin else 0.2, seed=5, permute=True)
    xyz = m.xyz if move is None else move(m)
    conn = np.ascontiguousarray(m.conn[:len(m.conn) - drop])
    kappa = meshgen.lognormal(len(conn), 1.0, 6)
    b = mg.MatrixBuilder(mg.Mesh(xyz, conn, order=1))
    _, rp, ci, ref = orc.full_operator(op, 1, 4, xyz, conn, coeff=kappa)
    room = torch.empty(len(kappa) + lead, dtype=torch.float64, device="cuda")
    coeff = room[lead:]
    coeff.copy_(torch.from_numpy(kappa))
    assert coeff.data_ptr() % 16 == 8 * lead
    v64 = b.assemble(op, coeff=coeff, quad=4, prec="f64").cpu().numpy()
    b.status()
    assert row_scaled_err(rp, ref, v64) <= F64_TOL
    if move is not _offset and move is not _thin:  # FP32 edges of ill-scaled meshes: not comparable at F32_TOL
        v32 = b.assemble(op, coeff=coeff, quad=4, prec="f32").cpu().numpy()
        assert row_scaled_err(rp, ref, v32) <= F32_TOL
