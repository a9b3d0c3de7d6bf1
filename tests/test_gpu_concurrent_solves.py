"""CG solves of different sizes on plans of their own, from two host threads on two
streams: each solve equals the one made alone, bit for bit.  The larger system takes
more shared memory than the smaller one and several launches."""
import threading

import numpy as np
import pytest

from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _system(n, sigma, seed):
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(n, jitter=0.2, seed=seed, permute=True)
    b = mg.MatrixBuilder(mg.Mesh(m.xyz, m.conn, order=1))
    A = b.assemble("stiff_kappa", coeff=meshgen.lognormal(len(m.conn), sigma, seed + 1), quad=4)
    b.apply_dirichlet(A, torch.from_numpy(m.boundary))
    x = np.random.default_rng(seed).uniform(-1.0, 1.0, b.ndof)
    return b, A, b.apply(A, torch.from_numpy(x).cuda())


@pytest.mark.parametrize("large,maxit", [(56, 4000), (34, 3000)])
def test_concurrent_cg_of_different_sizes(large, maxit):
    import torch
    big, small = _system(large, 3.0, 1), _system(6, 1.0, 2)
    kw = (dict(rtol=1e-14, maxit=maxit, precond=None, raise_on_fail=False), dict(rtol=1e-12))
    alone = [s[0].cg(s[1], s[2], **k)[0] for s, k in zip((big, small), kw)]
    torch.cuda.synchronize()
    errors, stop = [], threading.Event()

    def solve(system, which, repeat):
        b, A, rhs = system
        st = torch.cuda.Stream()
        try:
            with torch.cuda.stream(st):
                while repeat > 0 and not stop.is_set():
                    x, _ = b.cg(A, rhs, **kw[which])
                    st.synchronize()
                    if not torch.equal(x, alone[which]):
                        errors.append(f"system {which}: other values")
                    repeat -= 1
        except Exception as ex:  # reported to the main thread
            errors.append(repr(ex))

    other = threading.Thread(target=solve, args=(small, 1, 10 ** 6))
    other.start()
    solve(big, 0, 4)
    stop.set()
    other.join()
    assert not errors, errors[:3]
