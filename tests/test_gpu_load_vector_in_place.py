"""The load vector written over its own inputs: the same values as into an array of its own."""
import numpy as np
import pytest

from helpers import disjoint_tets
from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["one_pass", "isolated", "two_pass", "p2"])
def test_in_place(kind):
    import torch

    import morganapublic_gb300 as mg
    if kind == "two_pass":
        xyz, conn = disjoint_tets(700)
    else:
        m = meshgen.kuhn_cube(6 if kind == "p2" else 20, jitter=0.2, seed=2, permute=True)
        xyz, conn = m.xyz, m.conn
        if kind == "isolated":  # nodes outside every element
            conn = np.ascontiguousarray(conn[(conn < 5000).all(axis=1)])
    b = mg.MatrixBuilder(mg.Mesh(xyz, conn, order=2 if kind == "p2" else 1))
    rng = np.random.default_rng(4)
    f = torch.from_numpy(rng.uniform(-1, 1, b.ndof)).cuda()
    s = torch.from_numpy(rng.uniform(1, 2, len(conn))).cuda()
    want = b.build_vector(field=f, elem_scale=s)
    again = f.clone()
    assert torch.equal(b.build_vector(field=again, elem_scale=s, out=again), want)
    if len(conn) >= b.ndof:  # over the first values of the scale
        t = s.clone()
        assert torch.equal(b.build_vector(field=f, elem_scale=t, out=t[:b.ndof]), want)
    # one value into the field
    both = torch.cat([f, f[:1]])
    assert torch.equal(b.build_vector(field=both[:-1], elem_scale=s, out=both[1:]), want)
