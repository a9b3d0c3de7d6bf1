"""The first call of each kind on new handles, made on a non-blocking side stream: the
tables and row ranges it uploads are complete for that stream -- the same bits as on
the legacy stream."""
import numpy as np
import pytest

from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _first_calls(n, order, stream):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=n, permute=True)
    mesh = mg.Mesh(m.xyz, m.conn, order=order)
    b = mg.MatrixBuilder(mesh)
    mask = torch.from_numpy(m.boundary if order == 1 else meshgen.p2_boundary(m.boundary, mesh.edges()[0])).cuda()
    kappa = torch.from_numpy(meshgen.lognormal(len(m.conn), 1.0, n)).cuda()
    x = torch.from_numpy(np.random.default_rng(n).uniform(-1, 1, b.ndof)).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        rhs = b.build_vector(field=x, elem_scale=kappa, quad=4)
        A = b.assemble("stiff_kappa", coeff=kappa, quad=4 if order == 1 else 15)
        A32 = b.assemble("stiff_kappa", coeff=kappa, quad=4 if order == 1 else 15, prec="f32")
        lg = mg.LagrangeBuilder(b)
        B = lg.assemble(quad=3)
        S = lg.saddle(A, B)
        g = b.adjoint_grad(x, rhs, quad=4)
        b.apply_dirichlet(A, mask, rhs)
        b.apply_dirichlet(A32, mask)
        u, _ = b.cg(A, rhs, rtol=1e-10)
        v, _ = b.cg_refined(A, A32, rhs, rtol=1e-10)
    stream.synchronize()
    b.status()
    return [t.cpu() for t in (rhs, A, A32, B, S, g, u, v)]


@pytest.mark.parametrize("n,order", [(2, 1), (11, 1), (31, 1), (3, 2), (12, 2)])
def test_first_calls_on_a_side_stream(n, order):
    import torch
    want = _first_calls(n, order, torch.cuda.default_stream())
    for _ in range(3):
        got = _first_calls(n, order, torch.cuda.Stream())
        assert all(torch.equal(a, b) for a, b in zip(want, got))
