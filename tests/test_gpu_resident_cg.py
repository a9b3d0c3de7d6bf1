"""The resident CG (one cooperative kernel, systems that stay in L2) against the
three-kernel iteration, which mg_cg_solve_noalloc runs: one CTA, several, every
SM; rows longer than a pass; iteration limits, and more iterations than one launch
makes."""
import ctypes

import numpy as np
import pytest

from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _system(n, order, sigma, seed):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=seed, permute=True)
    mesh = mg.Mesh(m.xyz, m.conn, order=order)
    b = mg.MatrixBuilder(mesh)
    kappa = meshgen.lognormal(len(m.conn), sigma, seed + 1)
    mask = m.boundary if order == 1 else meshgen.p2_boundary(m.boundary, mesh.edges()[0])
    A = b.assemble("stiff_kappa", coeff=kappa, quad=4 if order == 1 else 11)
    b.apply_dirichlet(A, torch.from_numpy(mask))
    x = np.random.default_rng(seed).uniform(-1.0, 1.0, b.ndof)
    return b, kappa, mask, A, torch.from_numpy(x).cuda()


def _three_kernels(b, A, rhs, rtol, maxit, precond):
    import torch

    import morganapublic_gb300 as mg
    x, info = torch.zeros_like(rhs), mg.CgInfo()
    st = mg.lib().mg_cg_solve_noalloc(b._h, A.data_ptr(), rhs.data_ptr(), x.data_ptr(), rtol, maxit,
                                      mg.PRECOND[precond], ctypes.byref(info), torch.cuda.current_stream().cuda_stream)
    assert st in (mg.MG_OK, mg.MG_ERR_NOT_CONVERGED)
    return x, info


@pytest.mark.parametrize("n,order", [(2, 1), (5, 1), (6, 1), (17, 1), (34, 1), (2, 2), (9, 2)])
@pytest.mark.parametrize("precond", ["jacobi", None])
def test_resident_cg_matches_three_kernels(n, order, precond):
    b, _, _, A, u = _system(n, order, 1.0, 3 + n)
    rhs = b.apply(A, u)
    x, info = b.cg(A, rhs, rtol=1e-12, precond=precond)
    y, ref = _three_kernels(b, A, rhs, 1e-12, 10000, precond)
    assert info.converged and ref.converged
    assert abs(info.iterations - ref.iterations) <= 1 + ref.iterations // 50
    # both residuals are below 1e-12: the solutions agree to that times the condition
    assert float((x - y).norm() / u.norm()) <= 1e-8
    x2, _ = b.cg(A, rhs, rtol=1e-12, precond=precond)
    assert bool((x == x2).all())  # bitwise reproducible


@pytest.mark.parametrize("maxit", [1, 37, 511, 512, 513, 700])
def test_resident_cg_iteration_limit(maxit):
    # sigma 3 without a preconditioner: converges after about 860 iterations
    b, _, _, A, u = _system(14, 1, 3.0, 8)
    rhs = b.apply(A, u)
    x, info = b.cg(A, rhs, rtol=1e-14, maxit=maxit, precond=None, raise_on_fail=False)
    y, ref = _three_kernels(b, A, rhs, 1e-14, maxit, None)
    assert (info.iterations, info.converged) == (ref.iterations, ref.converged) == (maxit, 0)
    # later iterates of this system depend on the order of the sums (numpy's CG with two
    # orders: 7e-10 apart after 10 iterations, 3e-3 after 37)
    if maxit == 1:
        assert float((x - y).norm() / y.norm()) <= 1e-9


@pytest.mark.parametrize("n,order", [(5, 1), (20, 1), (9, 2)])
def test_resident_mixed_precision(n, order):
    import torch
    b, kappa, mask, A, u = _system(n, order, 1.0, 21 + n)
    A32 = b.assemble("stiff_kappa", coeff=kappa, quad=4 if order == 1 else 11, prec="f32")
    b.apply_dirichlet(A32, torch.from_numpy(mask))
    rhs = b.apply(A, u)
    x, info = b.cg_refined(A, A32, rhs, rtol=1e-11)
    assert info.converged and info.rel_residual <= 1e-11
    assert float((rhs - b.apply(A, x)).norm() / rhs.norm()) <= 1.5e-11
    assert float((x - u).norm() / u.norm()) <= 1e-7


def test_partition_outlives_a_larger_work_buffer():
    # the mixed-precision solve needs a larger work buffer than the FP64 one before it
    import torch
    b, kappa, mask, A, u = _system(9, 1, 1.0, 5)
    A32 = b.assemble("stiff_kappa", coeff=kappa, quad=4, prec="f32")
    b.apply_dirichlet(A32, torch.from_numpy(mask))
    rhs = b.apply(A, u)
    x, _ = b.cg(A, rhs, rtol=1e-10)
    b.cg_refined(A, A32, rhs, rtol=1e-10)
    filler = [torch.full((64,), 2**30, dtype=torch.int32, device="cuda") for _ in range(64)]
    y, _ = b.cg(A, rhs, rtol=1e-10)
    assert bool((x == y).all()) and len(filler) == 64
