"""Plans built on the GPU from packed coupling keys and shared scratch against
plans built on the host: dof counts at and around powers of two (the keys' width),
an unstructured numbering, and the arrays that outlive the scratch."""
import numpy as np
import pytest

from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,order", [(1, 1), (3, 1), (7, 1), (8, 1), (15, 1), (1, 2), (2, 2), (7, 2), (11, 2)])
def test_device_plan_matches_host_plan(n, order):
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.1, seed=n, permute=True)
    mesh = mg.Mesh(m.xyz, m.conn, order=order)
    host = mg.MatrixBuilder(mesh)
    built = mg.MatrixBuilder(mesh, pattern_on_device=True)
    for a, b in zip(built.pattern(), host.pattern()):
        assert np.array_equal(a, b)
    assert np.array_equal(built.elem_order(), host.elem_order())
    kappa = meshgen.lognormal(len(m.conn), 1.0, n)
    quad = 4 if order == 1 else 11
    want = host.assemble("stiff_kappa", coeff=kappa, quad=quad)
    # a second plan in between takes over the memory that the first one's build gave back
    other = mg.MatrixBuilder(mesh, pattern_on_device=True)
    got = built.assemble("stiff_kappa", coeff=kappa, quad=quad)
    assert bool((got == want).all())
    maps = "export_block_map" if order == 1 else "export_slot_map"
    a, b, c = (getattr(q, maps)() for q in (built, host, other))
    for k in b:
        assert np.array_equal(a[k], b[k]) and np.array_equal(c[k], b[k])


@pytest.mark.parametrize("order", [1, 2])
def test_nodes_without_elements_have_empty_rows(order):
    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(3, jitter=0.1, seed=2, permute=True)
    n = len(m.xyz)
    # unused nodes before, between and after the used ones
    place = np.arange(n) + 2 + 3 * (np.arange(n) >= n // 2)
    xyz = np.full((n + 9, 3), 0.5)
    xyz[place] = m.xyz
    mesh = mg.Mesh(xyz, place[m.conn].astype(np.int32), order=order)
    host, built = mg.MatrixBuilder(mesh), mg.MatrixBuilder(mesh, pattern_on_device=True)
    for a, b in zip(built.pattern(), host.pattern()):
        assert np.array_equal(a, b)
    rows = np.diff(built.pattern()[0])
    assert (rows[:n + 9] == 0).sum() == 9
    assert bool((built.assemble("mass") == host.assemble("mass")).all())


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("n", [510, 512, 513, 700])
def test_vertices_with_very_many_elements(n, order):
    # a fan: n elements around the edge between two vertices, whose rows the plan builds
    # by one thread each above 512 elements; against the oracle
    import oracle as orc
    from helpers import row_scaled_err

    import morganapublic_gb300 as mg
    angle = 2.0 * np.pi * np.arange(n) / n
    ring = np.stack([np.cos(angle), np.sin(angle), np.zeros(n)], axis=1)
    xyz = np.concatenate([ring, [[0.0, 0.0, -1.0], [0.0, 0.0, 1.0]]])
    i = np.arange(n)
    conn = np.stack([np.full(n, n), i, (i + 1) % n, np.full(n, n + 1)], axis=1).astype(np.int32)
    b = mg.MatrixBuilder(mg.Mesh(xyz, conn, order=order), pattern_on_device=True)
    kappa = meshgen.lognormal(n, 1.0, n)
    got = b.assemble("mass_coeff", coeff=kappa, quad=4).cpu().numpy()
    _, rp, ci, want = orc.full_operator("mass_coeff", order, 4, xyz, conn, coeff=kappa)
    rowptr, colind = b.pattern()
    assert np.array_equal(rowptr, rp) and np.array_equal(colind, ci)
    assert row_scaled_err(rp, want, got) <= 1e-12
