"""The finite-element operator path's workloads, as a user's program calls them.

Every case is a call (or the few calls that belong together) on a plan of a box
of Kuhn tetrahedra with jittered interior nodes and randomly permuted elements,
the mesh a program has after its mesher and partitioner:

    assemble  MatrixBuilder.assemble: CSR values of the listed operators
    spmv      MatrixBuilder.apply: y = A x
    cg        MatrixBuilder.cg: Jacobi-PCG in FP64
    refined   MatrixBuilder.cg_refined: FP32 iteration, FP64 residuals
    vector    MatrixBuilder.build_vector: the load vector
    adjoint   MatrixBuilder.adjoint_grad: dJ/dkappa per element
    boundary  LagrangeBuilder.assemble and .saddle: B and [K B^T; B 0]
    build     host arrays -> Mesh -> MatrixBuilder -> build_crs: host CSR

Inputs are made on the GPU from the seed alone.
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

import morganapublic_gb300 as mg

EDGES = ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))  # local edges of the P2 basis
FACES = ((0, 2, 1), (0, 1, 3), (1, 2, 3), (0, 3, 2))


def _case(name, kind, nx, ny, nz, order=1, prec="f64", ops="stiff_kappa", jitter=0.2, sigma=1.0):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "order": order, "prec": prec, "ops": ops,
            "jitter": jitter, "sigma": sigma}


def listed():
    return [
        # the 128^3 diffusion operator of the headline benchmark, re-assembled as kappa changes
        _case("assemble_p1_f64_128", "assemble", 128, 128, 128, jitter=0.25, sigma=1.5),
        # the FP32 operator of a mixed-precision solve, at 64^3
        _case("assemble_p1_f32_64", "assemble", 64, 64, 64, prec="f32"),
        # Laplace stiffness and consistent mass of a small problem (16^3): launch latency
        _case("assemble_p1_small", "assemble", 16, 16, 16, ops="stiff_const+mass", jitter=0.1),
        # the quadratic element's diffusion operator, 48^3
        _case("assemble_p2_f64_48", "assemble", 48, 48, 48, order=2, sigma=0.5),
        # one product of a Krylov loop that the user's own solver runs, 128^3
        _case("spmv_p1_f64_128", "spmv", 128, 128, 128, jitter=0.25, sigma=1.5),
        # the same on quadratic elements in FP32, on a box with odd sides
        _case("spmv_p2_f32_ragged", "spmv", 37, 51, 43, order=2, prec="f32", sigma=0.5),
        # a forward solve, 64^3
        _case("cg_p1_64", "cg", 64, 64, 64),
        # a mixed-precision solve on quadratic elements, 48^3
        _case("refined_p2_48", "refined", 48, 48, 48, order=2, sigma=0.5),
        # the right-hand side of a time step (nodal field, element scale), 96^3
        _case("vector_p1_96", "vector", 96, 96, 96),
        # the gradient of an inversion step, 64^3
        _case("adjoint_p1_64", "adjoint", 64, 64, 64, sigma=0.5),
        # Dirichlet data by boundary multipliers: B and the saddle matrix, odd sides
        _case("boundary_p1_ragged", "boundary", 41, 47, 35),
        # a new mesh: from host arrays to the host CSR matrix, 64^3
        _case("build_p1_64", "build", 64, 64, 64),
    ]


# cells of the largest drawn mesh, by kind and order (at most the listed ones' cost)
MOST_CELLS = {("assemble", 1): 128**3, ("assemble", 2): 48**3, ("spmv", 1): 128**3, ("spmv", 2): 48**3,
              ("cg", 1): 64**3, ("cg", 2): 24**3, ("refined", 1): 64**3, ("refined", 2): 48**3,
              ("vector", 1): 96**3, ("vector", 2): 48**3, ("adjoint", 1): 64**3, ("adjoint", 2): 32**3,
              ("boundary", 1): 41 * 47 * 35, ("boundary", 2): 20**3, ("build", 1): 64**3, ("build", 2): 24**3}


def draw(rng):
    kind = rng.choice(("assemble", "assemble", "spmv", "spmv", "cg", "refined", "vector", "adjoint", "boundary", "build"))
    order = rng.choice((1, 1, 2))
    cells = math.exp(rng.uniform(math.log(7**3), math.log(MOST_CELLS[kind, order])))
    side = cells ** (1.0 / 3.0)
    a, b = math.exp(rng.uniform(-0.4, 0.4)), math.exp(rng.uniform(-0.4, 0.4))
    nx, ny = max(3, round(side * a)), max(3, round(side * b))
    nz = max(3, int(cells / (nx * ny)))
    while nx * ny * nz > MOST_CELLS[kind, order]:
        nx, ny, nz = (n - 1 if n == max(nx, ny, nz) else n for n in (nx, ny, nz))
    prec = rng.choice(("f64", "f32")) if kind in ("assemble", "spmv") else "f64"
    ops = rng.choice(("stiff_kappa", "stiff_kappa", "mass_coeff", "stiff_const+mass")) if kind == "assemble" else "stiff_kappa"
    c = _case("", kind, nx, ny, nz, order=order, prec=prec, ops=ops, jitter=rng.choice((0.05, 0.1, 0.2, 0.25)),
              sigma=rng.choice((0.0, 0.5, 1.0, 1.5)))
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs --
def _kuhn():
    """Six tetrahedra of the unit cell as corner numbers 4 i + 2 j + k, each positively oriented."""
    tets = []
    for axes in itertools.permutations(range(3)):
        v, pts = [0, 0, 0], [(0, 0, 0)]
        for a in axes:
            v[a] = 1
            pts.append(tuple(v))
        if np.linalg.det(np.array([np.subtract(p, pts[0]) for p in pts[1:]], dtype=float)) < 0:
            pts[2], pts[3] = pts[3], pts[2]
        tets.append([4 * p[0] + 2 * p[1] + p[2] for p in pts])
    return tets


def _edge_vectors(xyz, conn):
    x0 = xyz[conn[:, 0]]
    return torch.stack([xyz[conn[:, k]] - x0 for k in (1, 2, 3)], dim=2)  # J[e, :, k]


def _dets(xyz, conn):
    J = _edge_vectors(xyz, conn)
    return (J[:, :, 0] * torch.linalg.cross(J[:, :, 1], J[:, :, 2])).sum(1)


def _mesh(case, seed):
    """(xyz (N, 3) float64, conn (E, 4) int64, boundary (N,) bool, generator), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    nx, ny, nz, jitter = case["nx"], case["ny"], case["nz"], case["jitter"]
    h = 1.0 / max(nx, ny, nz)
    ar = lambda n: torch.arange(n, device="cuda")  # noqa: E731
    ijk = torch.stack(torch.meshgrid(ar(nx + 1), ar(ny + 1), ar(nz + 1), indexing="ij"), -1).reshape(-1, 3)
    top = torch.tensor([nx, ny, nz], device="cuda")
    boundary = ((ijk == 0) | (ijk == top)).any(1)
    base = ijk.double() * h
    cell = torch.stack(torch.meshgrid(ar(nx), ar(ny), ar(nz), indexing="ij"), -1).reshape(-1, 3)
    first = (cell[:, 0] * (ny + 1) + cell[:, 1]) * (nz + 1) + cell[:, 2]
    corner = torch.tensor([((c >> 2) * (ny + 1) + ((c >> 1) & 1)) * (nz + 1) + (c & 1) for c in range(8)], device="cuda")
    conn = (first[:, None, None] + corner[torch.tensor(_kuhn(), device="cuda")][None]).reshape(-1, 4)
    move = lambda: (torch.rand(base.shape, dtype=torch.float64, device="cuda", generator=g) * 2 - 1) * (jitter * h)  # noqa: E731
    xyz = base
    if jitter > 0:
        xyz = torch.where(boundary[:, None], base, base + move())
        for _ in range(64):  # new positions for the nodes of a tetrahedron that came out inverted
            bad = _dets(xyz, conn) <= 1e-3 * h**3
            if not bool(bad.any()):
                break
            at = torch.zeros(len(xyz), dtype=torch.bool, device="cuda")
            at[conn[bad].reshape(-1)] = True
            xyz = torch.where((at & ~boundary)[:, None], base + move(), xyz)
    conn = conn[torch.randperm(len(conn), device="cuda", generator=g)]
    return xyz.contiguous(), conn.contiguous(), boundary, g


def _kappa(case, E, g):
    return torch.exp(case["sigma"] * torch.randn(E, dtype=torch.float64, device="cuda", generator=g))


def _uniform(n, g, dtype=torch.float64):
    return (torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1).to(dtype)


def _dofs(case, conn, n_nodes):
    """Element dofs (E, 4 or 10) and the nodes of the P2 edges in dof order (min, max)."""
    if case["order"] == 1:
        return conn, None
    a = torch.tensor(EDGES, device="cuda")
    p, q = conn[:, a[:, 0]], conn[:, a[:, 1]]
    key = torch.minimum(p, q) * n_nodes + torch.maximum(p, q)
    edges, at = torch.unique(key, return_inverse=True)
    return torch.cat([conn, n_nodes + at], 1), torch.stack([edges // n_nodes, edges % n_nodes], 1)


def _points(xyz, edges):
    return xyz if edges is None else torch.cat([xyz, 0.5 * (xyz[edges[:, 0]] + xyz[edges[:, 1]])])


def _field(X, g):
    """A smooth field with some noise: a state, an adjoint state, a source."""
    k = 3.0 + 2.0 * _uniform(3, g)
    return torch.sin(X @ k) + X[:, 0] * X[:, 1] + 0.05 * _uniform(len(X), g)


def _state(case, X, g):
    """A solution of the Dirichlet problem with zero boundary data: a few sine modes of the box."""
    top = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device="cuda")
    Y = X * (math.pi * float(top.max()) / top)
    return sum(c * torch.sin(Y[:, 0] * (k & 1 or 2)) * torch.sin(Y[:, 1] * (k & 2 or 1)) * torch.sin(Y[:, 2] * (k // 4 + 1)) for k, c in enumerate(1.0 + _uniform(8, g)))


def _quad(case):
    return 4 if case["order"] == 1 else 11


def _everything(case, seed):
    xyz, conn, boundary, g = _mesh(case, seed)
    s = {"case": case, "xyz": xyz, "conn": conn, "boundary": boundary, "kappa": _kappa(case, len(conn), g)}
    s["dofs"], s["edges"] = _dofs(case, conn, len(xyz))
    s["ndof"] = len(xyz) if s["edges"] is None else len(xyz) + len(s["edges"])
    X = _points(xyz, s["edges"])
    if case["kind"] == "spmv":
        s["x"] = _uniform(s["ndof"], g, torch.float64 if case["prec"] == "f64" else torch.float32)
    elif case["kind"] in ("cg", "refined"):
        s["u"] = _state(case, X, g)
    elif case["kind"] == "vector":
        s["f"] = _field(X, g)
    elif case["kind"] == "adjoint":
        s["u"], s["lam"] = _field(X, g), _field(X, g)
    return s


def prepare(case, seed):
    if case["kind"] == "build":  # the program has a mesh and a coefficient on the host
        xyz, conn, _, g = _mesh(case, seed)
        return {"case": case, "xyz": xyz.cpu().numpy(), "conn": conn.int().cpu().numpy(), "kappa": _kappa(case, len(conn), g).cpu().numpy()}
    s = _everything(case, seed)
    mesh = mg.Mesh(s["xyz"].cpu().numpy(), s["conn"].int().cpu().numpy(), order=case["order"], edges_on_device=case["order"] == 2)
    b = mg.MatrixBuilder(mesh, pattern_on_device=True)
    st = {"case": case, "mesh": mesh, "b": b, "kappa": s["kappa"]}
    quad, kind = _quad(case), case["kind"]
    if kind == "assemble":  # the program's value arrays, filled again on each call
        dt = torch.float64 if case["prec"] == "f64" else torch.float32
        st["out"] = [torch.empty(b.nnz, dtype=dt, device="cuda") for _ in case["ops"].split("+")]
    elif kind == "spmv":
        st["A"] = b.assemble("stiff_kappa", coeff=s["kappa"], quad=quad, prec=case["prec"])
        st["x"], st["y"] = s["x"], torch.empty_like(s["x"])
    elif kind in ("cg", "refined"):
        edges, mask = s["edges"], s["boundary"]
        if edges is not None:
            mask = torch.cat([mask, mask[edges[:, 0]] & mask[edges[:, 1]]])
        st["A"] = b.assemble("stiff_kappa", coeff=s["kappa"], quad=quad)
        b.apply_dirichlet(st["A"], mask)
        if kind == "refined":
            st["A32"] = b.assemble("stiff_kappa", coeff=s["kappa"], quad=quad, prec="f32")
            b.apply_dirichlet(st["A32"], mask)
        st["rhs"] = b.apply(st["A"], s["u"])  # so that u is the discrete solution
    elif kind == "vector":
        st["f"], st["out"] = s["f"], torch.empty(b.ndof, dtype=torch.float64, device="cuda")
    elif kind == "adjoint":
        st["u"], st["lam"] = s["u"], s["lam"]
        st["out"] = torch.empty(mesh.n_elements, dtype=torch.float64, device="cuda")
    else:
        st["K"] = b.assemble("stiff_kappa", coeff=s["kappa"], quad=quad)
        st["L"] = mg.LagrangeBuilder(b)
        st["B"] = torch.empty(st["L"].nnz_b, dtype=torch.float64, device="cuda")
        st["S"] = torch.empty(st["L"].nnz_saddle, dtype=torch.float64, device="cuda")
    return st


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    quad = _quad(case)
    if kind == "assemble":
        return [s["b"].assemble(op, coeff=s["kappa"], quad=quad, prec=case["prec"], out=out) for op, out in zip(case["ops"].split("+"), s["out"])]
    if kind == "spmv":
        return s["b"].apply(s["A"], s["x"], out=s["y"])
    if kind == "cg":
        return s["b"].cg(s["A"], s["rhs"], rtol=1e-10)[0]
    if kind == "refined":
        return s["b"].cg_refined(s["A"], s["A32"], s["rhs"], rtol=1e-10)[0]
    if kind == "vector":
        return s["b"].build_vector(field=s["f"], elem_scale=s["kappa"], quad=quad, out=s["out"])
    if kind == "adjoint":
        return s["b"].adjoint_grad(s["u"], s["lam"], quad=quad, out=s["out"])
    if kind == "boundary":
        B = s["L"].assemble(quad=3 if case["order"] == 1 else 6, out=s["B"])
        return {"B": B, "S": s["L"].saddle(s["K"], B, out=s["S"])}
    mesh = mg.Mesh(s["xyz"], s["conn"], order=case["order"], edges_on_device=case["order"] == 2)
    b = mg.MatrixBuilder(mesh, pattern_on_device=True)
    a = b.build_crs("stiff_kappa", coeff=s["kappa"], quad=quad)
    b.close()
    mesh.close()
    return {"rowptr": a.rowptr, "colind": a.colind, "values": a.values}


# --------------------------------------------------------------------- work --
def _sizes(case):
    """Elements, nodes, dofs, CSR entries and boundary triangles of the box."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    E, N = 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    edges = 0
    for a, b, c in itertools.product((0, 1), repeat=3):  # an edge along each nonzero corner of the cell
        if a + b + c:
            edges += (nx + 1 - a) * (ny + 1 - b) * (nz + 1 - c)
    F = 4 * (nx * ny + ny * nz + nz * nx)
    if case["order"] == 1:
        return E, N, N, N + 2 * edges, F
    tri = (4 * E + F) // 2
    return E, N, N + edges, (N + 2 * edges) + 2 * (2 * edges + 3 * tri) + (edges + 6 * tri + 6 * E), F


def work(case):
    E, N, nd, nnz, F = _sizes(case)
    kind, nb = case["kind"], 4 if case["order"] == 1 else 10
    sv = 8 if case["prec"] == "f64" else 4
    per_elem = 16 + 4 * (nb - 4)  # connectivity and further dofs
    stiff_flops = 130 if nb == 4 else 800
    if kind == "assemble":  # connectivity, coefficient and coordinates in, values out
        n = len(case["ops"].split("+"))
        one = E * (per_elem + (8 if "const" not in case["ops"] else 0)) + 24 * N + sv * nnz
        return {"bytes": n * one, "flops": n * E * stiff_flops}
    spmv = nnz * (sv + 4) + 4 * (nd + 1) + 2 * sv * nd
    if kind == "spmv":
        return {"bytes": spmv, "flops": 2 * nnz}
    if kind in ("cg", "refined"):  # about 7.7 (P1) or 10 (P2) iterations per cell of the longest side
        its = (7.7 if nb == 4 else 10.0) * max(case["nx"], case["ny"], case["nz"])
        if kind == "refined":
            return {"bytes": its * (nnz * 8 + 4 * nd + 12 * 4 * nd), "flops": its * (2 * nnz + 12 * nd)}
        return {"bytes": its * (spmv + 12 * 8 * nd), "flops": its * (2 * nnz + 12 * nd)}
    if kind == "vector":
        return {"bytes": E * (per_elem + 8) + 24 * N + 16 * nd, "flops": E * (50 + 2 * nb * nb)}
    if kind == "adjoint":
        return {"bytes": E * (per_elem + 8) + 24 * N + 16 * nd, "flops": E * (80 if nb == 4 else 900)}
    if kind == "boundary":  # faces in, B out; K in and the saddle matrix (K, B, B^T) out
        nnz_b = 9 * F // 2 * (1 if nb == 4 else 3)
        return {"bytes": F * 20 + 8 * nnz_b + 16 * nnz + 8 * 3 * nnz_b, "flops": F * 300}
    return {"bytes": E * (per_elem + 8) + 24 * N + 12 * nnz + 4 * nd, "flops": E * stiff_flops}


# -------------------------------------------------------------------- exact --
def _duffy(dim, n=6):
    """Points and weights of the reference simplex, exact beyond every integrand here."""
    t, w = np.polynomial.legendre.leggauss(n)
    t, w = (t + 1) / 2, w / 2
    pts, wts = [], []
    for ix in itertools.product(range(n), repeat=dim):
        rest, p, ww = 1.0, [], 1.0
        for d, i in enumerate(ix):
            ww *= w[i] * rest
            p.append(t[i] * rest)
            rest *= 1 - t[i]
        pts.append(p)
        wts.append(ww)
    return np.array(pts), np.array(wts)


def _basis(order, L):
    """phi (points, nb) for barycentric L (points, 4)."""
    if order == 1:
        return L
    return np.concatenate([L * (2 * L - 1), np.stack([4 * L[:, a] * L[:, b] for a, b in EDGES], 1)], 1)


def _tables(order):
    """S[a, b, i, j] = int d_a phi_i d_b phi_j and M[i, j] = int phi_i phi_j over the reference tetrahedron."""
    p, w = _duffy(3)
    L = np.concatenate([1 - p.sum(1, keepdims=True), p], 1)
    G = np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=float)  # grad of L
    if order == 1:
        dphi = np.broadcast_to(G, (len(p), 4, 3))
    else:
        dphi = np.concatenate([(4 * L - 1)[:, :, None] * G, np.stack([4 * (L[:, a, None] * G[b] + L[:, b, None] * G[a]) for a, b in EDGES], 1)], 1)
    phi = _basis(order, L)
    dev = lambda a: torch.tensor(a, device="cuda")  # noqa: E731
    return dev(np.einsum("q,qia,qjb->abij", w, dphi, dphi)), dev(np.einsum("q,qi,qj->ij", w, phi, phi))


def _cofactors(xyz, conn):
    """C (E, 3, 3) with column a the cofactor column of J, and det J."""
    J = _edge_vectors(xyz, conn)
    C = torch.stack([torch.linalg.cross(J[:, :, (a + 1) % 3], J[:, :, (a + 2) % 3]) for a in range(3)], 2)
    return C, (J[:, :, 0] * C[:, :, 0]).sum(1)


def _element_matrices(s, op, lo, hi):
    S, M = _tables(s["case"]["order"])
    C, det = _cofactors(s["xyz"], s["conn"][lo:hi])
    kap = s["kappa"][lo:hi] if op in ("stiff_kappa", "mass_coeff") else torch.ones_like(det)
    if op.startswith("stiff"):
        return torch.einsum("eab,abij->eij", torch.einsum("era,erb->eab", C, C) * (kap / det)[:, None, None], S)
    return M[None] * (kap * det)[:, None, None]


def _csr(s, ops):
    """(row * ndof + col keys in CSR order, values of each operator)."""
    dofs, nd = s["dofs"], s["ndof"]
    nb = dofs.shape[1]
    key = (dofs[:, :, None] * nd + dofs[:, None, :]).reshape(-1)
    keys, at = torch.unique(key, return_inverse=True)
    del key
    vals, step = [], 1 << 20
    for op in ops:
        v = torch.zeros(len(keys), dtype=torch.float64, device="cuda")
        for lo in range(0, len(dofs), step):
            K = _element_matrices(s, op, lo, min(len(dofs), lo + step))
            v.index_add_(0, at[lo * nb * nb:(lo + len(K)) * nb * nb], K.reshape(-1))
        vals.append(v)
    return keys, vals


def _boundary_exact(s):
    """B and the saddle matrix, both in CSR order."""
    conn, dofs, nd, order = s["conn"], s["dofs"], s["ndof"], s["case"]["order"]
    n = len(s["xyz"])
    tri = torch.stack([torch.sort(conn[:, list(f)], 1)[0] for f in FACES], 1)  # (E, 4, 3)
    code = (tri[..., 0] * n + tri[..., 1]) * n + tri[..., 2]
    _, at, count = torch.unique(code, return_inverse=True, return_counts=True)
    elem, local = torch.nonzero(count[at] == 1, as_tuple=True)
    p, w = _duffy(2)
    lam = np.concatenate([1 - p.sum(1, keepdims=True), p], 1)
    T = []
    for f in FACES:
        L = np.zeros((len(p), 4))
        L[:, list(f)] = lam
        T.append(np.einsum("q,qa,qi->ai", w, lam, _basis(order, L)))
    T = torch.tensor(np.array(T), device="cuda")
    nodes = torch.gather(conn[elem], 1, torch.tensor(FACES, device="cuda")[local])  # (F, 3)
    X = s["xyz"][nodes]
    area2 = torch.linalg.cross(X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]).norm(dim=1)
    lam_nodes, row = torch.unique(nodes, return_inverse=True)
    key = (row[:, :, None] * nd + dofs[elem][:, None, :]).reshape(-1)
    bkeys, at = torch.unique(key, return_inverse=True)
    B = torch.zeros(len(bkeys), dtype=torch.float64, device="cuda")
    B.index_add_(0, at, (T[local] * area2[:, None, None]).reshape(-1))
    keys, (K,) = _csr(s, ("stiff_kappa",))
    full = nd + len(lam_nodes)
    bl, bc = bkeys // nd, bkeys % nd
    order_of = torch.cat([keys // nd * full + keys % nd, bc * full + nd + bl, (nd + bl) * full + bc])
    return {"B": B, "S": torch.cat([K, B, B])[torch.argsort(order_of)]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "build":
        xyz, conn, boundary, g = _mesh(case, seed)
        s = {"case": case, "xyz": xyz, "conn": conn, "kappa": _kappa(case, len(conn), g)}
        s["dofs"], s["edges"] = _dofs(case, conn, len(xyz))
        s["ndof"] = len(xyz) if s["edges"] is None else len(xyz) + len(s["edges"])
        return {"rowptr": None, "colind": None, "values": _csr(s, ("stiff_kappa",))[1][0]}
    s = _everything(case, seed)
    if kind == "assemble":
        return _csr(s, case["ops"].split("+"))[1]
    if kind == "spmv":
        keys, (v,) = _csr(s, ("stiff_kappa",))
        y = torch.zeros(s["ndof"], dtype=torch.float64, device="cuda")
        return y.index_add_(0, keys // s["ndof"], v * s["x"].double()[keys % s["ndof"]])
    if kind in ("cg", "refined"):
        return s["u"]
    if kind == "boundary":
        return _boundary_exact(s)
    S, M = _tables(case["order"])
    C, det = _cofactors(s["xyz"], s["conn"])
    dofs = s["dofs"]
    if kind == "vector":
        y = (s["f"][dofs] @ M) * (s["kappa"] * det)[:, None]
        return torch.zeros(s["ndof"], dtype=torch.float64, device="cuda").index_add_(0, dofs.reshape(-1), y.reshape(-1))
    u, lam = (s[k][dofs] - s[k][dofs[:, :1]] for k in ("u", "lam"))  # the form only sees differences
    m = torch.einsum("era,erb->eab", C, C) / det[:, None, None]
    return -torch.einsum("eab,ei,ej,abij->e", m, u, lam, S)
