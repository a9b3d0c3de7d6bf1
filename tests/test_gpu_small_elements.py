"""Elements very small beside the mesh: edges exact to the double-word arithmetic at
every ratio of sizes -- assembly and load vector against the oracle."""
import numpy as np
import pytest

import oracle as orc
from helpers import row_scaled_err

pytestmark = pytest.mark.gpu


def _mesh(ratio):
    """A tetrahedron of 2^30 and four of 2^(30 + ratio) with full mantissas near the origin."""
    rng = np.random.default_rng(11)
    ref = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=np.float64)
    size = 2.0 ** (30 + ratio)
    parts = [2.0 ** 30 * (ref + 0.1 * rng.uniform(-1, 1, (4, 3)))]
    parts += [size * (ref + 0.1 * rng.uniform(-1, 1, (4, 3)) + rng.uniform(-1, 1, 3)) for _ in range(4)]
    xyz = np.concatenate(parts)
    return xyz, np.arange(len(xyz), dtype=np.int32).reshape(-1, 4)


@pytest.mark.parametrize("ratio", [-10, -19, -22, -30, -36, -38, -41, -44, -47, -50, -55])
@pytest.mark.parametrize("op,order,quad", [("stiff_kappa", 1, 4), ("mass_coeff", 1, 4), ("stiff_kappa", 2, 15)])
def test_small_elements_match_oracle(ratio, op, order, quad):
    import morganapublic_gb300 as mg
    xyz, conn = _mesh(ratio)
    kappa = np.random.default_rng(2).uniform(0.5, 2.0, len(conn))
    b = mg.MatrixBuilder(mg.Mesh(xyz, conn, order=order))
    _, rp, ci, ref = orc.full_operator(op, order, quad, xyz, conn, coeff=kappa)
    got = b.assemble(op, coeff=kappa, quad=quad).cpu().numpy()
    b.status()
    assert row_scaled_err(rp, ref, got) <= 1e-12
    if order == 1:
        v = b.build_vector(elem_scale=kappa, quad=quad).cpu().numpy()
        vref = orc.assemble_rhs(1, quad, xyz, conn, conn, len(xyz), elem_scale=kappa)
        assert np.max(np.abs(v - vref) / np.abs(vref)) <= 1e-12
