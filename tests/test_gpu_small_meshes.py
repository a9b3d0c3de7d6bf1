"""Very small meshes (edges of 1e-6 to 1e-14): stiffness, mass, load vector and adjoint as
accurate as at any size, and the same bits as on the mesh times a power of two."""
import numpy as np
import pytest

import oracle as orc
from helpers import disjoint_tets, row_scaled_err
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _setup(n, order, size):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=3, permute=True)
    xyz = m.xyz * size
    b = mg.MatrixBuilder(mg.Mesh(xyz, m.conn, order=order))
    rng = np.random.default_rng(n)
    kappa = np.exp(rng.normal(size=len(m.conn)))
    u, v = (torch.from_numpy(rng.uniform(-1, 1, b.ndof)).cuda() for _ in range(2))
    return m, xyz, b, kappa, u, v


@pytest.mark.parametrize("order,quad", [(1, 4), (2, 15)])
@pytest.mark.parametrize("h", [1e-3, 1e-6, 1e-8, 1e-9, 1e-10, 1e-12, 1e-14])
def test_small_mesh_matches_oracle(order, quad, h):
    import morganapublic_gb300 as mg
    n = 7
    m, xyz, b, kappa, u, v = _setup(n, order, n * h)
    dofs, rp, ci, ref = orc.full_operator("stiff_kappa", order, quad, xyz, m.conn, coeff=kappa)
    assert row_scaled_err(rp, ref, b.assemble("stiff_kappa", coeff=kappa, quad=quad).cpu().numpy()) <= 1e-12
    assert row_scaled_err(rp, ref, b.assemble("stiff_kappa", coeff=kappa, quad=quad, prec="f32").cpu().numpy()) <= 2e-6
    b.status()
    g = orc.adjoint_grad(order, quad, xyz, m.conn, dofs, u.cpu().numpy(), v.cpu().numpy())
    assert np.max(np.abs(b.adjoint_grad(u, v, quad=quad).cpu().numpy() - g)) <= 1e-12 * np.abs(g).max()
    f = np.abs(u.cpu().numpy()) + 0.5
    r = orc.assemble_rhs(order, quad, xyz, m.conn, dofs, b.ndof, field=f, elem_scale=kappa)
    size = orc.assemble_rhs(order, quad, xyz, m.conn, dofs, b.ndof)  # of the entries (P2: of both signs)
    got = b.build_vector(field=f, elem_scale=kappa, quad=quad).cpu().numpy()
    assert np.all(np.abs(got - r) <= 1e-12 * np.abs(kappa).max() * np.abs(size).max())
    # determinants of h^3: the values leave the double-words below h of about 1e-10
    _, _, _, ref = orc.full_operator("mass_coeff", order, quad, xyz, m.conn, coeff=kappa)
    got = b.assemble("mass_coeff", coeff=kappa, quad=quad).cpu().numpy()
    if h < 5e-10:
        with pytest.raises(mg.MorganaError):
            b.status()
    else:
        b.status()
        assert row_scaled_err(rp, ref, got) <= 1e-12
    # entries that are normal floats: 1e12 h^3 for h down to 1e-14
    _, _, _, ref = orc.full_operator("mass_coeff", order, quad, xyz, m.conn, coeff=kappa * 1e12)
    got = b.assemble("mass_coeff", coeff=kappa * 1e12, quad=quad, prec="f32").cpu().numpy()
    assert row_scaled_err(rp, ref, got) <= 2e-6


@pytest.mark.parametrize("order,quad", [(1, 4), (2, 15)])
@pytest.mark.parametrize("k", [-6, -9, -10, -24, -40])
def test_power_of_two_of_a_mesh(order, quad, k):
    m, _, b, kappa, u, v = _setup(6, order, 1.0)
    _, _, c, _, _, _ = _setup(6, order, 2.0 ** k)
    for prec in ("f64", "f32"):
        x = b.assemble("stiff_kappa", coeff=kappa, quad=quad, prec=prec).double()
        y = c.assemble("stiff_kappa", coeff=kappa, quad=quad, prec=prec).double()
        assert bool((x * 2.0 ** k == y).all())
        if k >= -24:
            x = b.assemble("mass_coeff", coeff=kappa, quad=quad, prec=prec).double()
            y = c.assemble("mass_coeff", coeff=kappa, quad=quad, prec=prec).double()
            assert bool((x * 2.0 ** (3 * k) == y).all())
    c.status()
    for f, s in ((u, kappa), (None, None), (u * 1e-300, kappa * 1e-8), (u * 10.0 ** (-100 * u), kappa)):
        x, y = (p.build_vector(field=f, elem_scale=s, quad=quad) for p in (b, c))
        # exact but for results below the normal doubles
        assert bool(((x * 2.0 ** (3 * k) - y).abs() <= 24 * 2.0 ** -1074).all())
    x, y = (p.adjoint_grad(u, v, quad=quad) for p in (b, c))
    assert bool((x * 2.0 ** k == y).all())


def test_small_mesh_two_pass_vector():
    import torch

    import morganapublic_gb300 as mg
    xyz, conn = disjoint_tets(700)
    f = torch.from_numpy(np.random.default_rng(1).uniform(1, 2, len(xyz))).cuda()
    x, y = (mg.MatrixBuilder(mg.Mesh(xyz * s, conn, order=1)).build_vector(field=f, quad=4) for s in (1.0, 2.0 ** -33))
    assert bool((x * 2.0 ** -99 == y).all())
