"""What is measured: the calls a user of this framework makes, over the sizes they make them at.

Six kinds of pass, each through the public entry point that a program calls:

* ``assemble``: E and B of a mesh on the device (``CsrPlan.assemble``), the step of every sweep, material
  study or optimisation loop that changes the tensors; the plan (symbolic phase) is kept per mesh.
* ``drop_in``:  the reference's own call, ``tet_mass_stiffness_matrices``: host tensors in, SciPy CSR out.
* ``apply``:    K_f x for a batch of systems (``FrequencySweep.apply``): residual checks, own iterations.
* ``sweep``:    the batched Krylov frequency sweep (``FrequencySweep.solve``).
* ``lu`` / ``direct``: the direct solve, as factor + solve of one frequency (``DeviceLU``) and as a window of
  neighbouring frequencies (``FrequencySweep.solve_direct``).
* ``network``:  one training pass of the preconditioner's network, forward and backward.

Meshes are the repository's seeded box families (guide, cavity, substrate); ``exact`` restates the
element, boundary and network formulas in plain torch at 64 bits and solves densely.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from emerge_b200 import problems
from emerge_b200.assembly import CsrPlan, DeviceMesh, tet_mass_stiffness_matrices
from emerge_b200.auxspace import AuxSpace, Network
from emerge_b200.sweep import FrequencySweep

C0, Z0 = 299792458.0, 376.73031366857


# ------------------------------------------------------------------------------------------ cases
def listed() -> list[dict]:
    return [
        # the 6 000-tet air-filled guide: the smallest mesh in use, launches and latency count
        dict(name="assemble_guide_6k", kind="assemble", family="guide", nx=10, ny=5, nz=20, materials="air"),
        # the benchmark mesh, 40^3 x 6 = 384 000 tets, lossy dielectric blocks
        dict(name="assemble_cavity_384k", kind="assemble", family="cavity", nx=40, ny=40, nz=40, materials="blocks"),
        # a ragged grid with every local orientation and full complex tensors, host to host
        dict(name="drop_in_ragged_tensor", kind="drop_in", family="guide", nx=17, ny=11, nz=13, materials="tensor"),
        # one system's operator on the small guide: the smallest call of the solve path
        dict(name="apply_guide_1", kind="apply", family="guide", nx=10, ny=5, nz=20, materials="air", nsys=1),
        # 16 systems on an 82 944-tet cavity: beyond L2
        dict(name="apply_cavity_16", kind="apply", family="cavity", nx=24, ny=24, nz=24, materials="blocks", nsys=16),
        # the guide sweep of the benchmark: 16 frequencies x 2 ports in one batch, aux-space correction
        dict(name="sweep_aux_guide_32", kind="sweep", family="guide", nx=10, ny=5, nz=20, materials="air",
             nfreq=16, nport=2, precond="aux", precision="fp64"),
        # FP32 inner iterations in FP64 refinement, an odd batch
        dict(name="sweep_mixed_guide_7", kind="sweep", family="guide", nx=8, ny=4, nz=11, materials="air",
             nfreq=7, nport=1, precond="aux", precision="mixed"),
        # the default preconditioner on a very small mesh: a chain of short kernels
        dict(name="sweep_plain_small_4", kind="sweep", family="guide", nx=5, ny=3, nz=9, materials="air",
             nfreq=2, nport=2, precond="block_jacobi", precision="fp64"),
        # the direct solve of one frequency of an 82 944-tet cavity: factor, then 8 right-hand sides
        dict(name="lu_cavity_24", kind="lu", family="cavity", nx=24, ny=24, nz=24, materials="blocks", nrhs=8),
        # a window of 9 neighbouring frequencies from one complex64 factorization
        dict(name="direct_cavity_window_9", kind="direct", family="cavity", nx=16, ny=16, nz=16, materials="blocks",
             nfreq=9, nport=1, precision="c64"),
        # low frequency on a substrate box: complex128 fronts, both lumped ports
        dict(name="direct_substrate_c128", kind="direct", family="substrate", nx=11, ny=8, nz=7, materials="layer",
             nfreq=2, nport=2, precision="c128"),
        # one training pass of the learned preconditioner on the guide, 8 right-hand sides
        dict(name="network_train_guide_8", kind="network", family="guide", nx=10, ny=5, nz=20, materials="air",
             nsys=8),
    ]


def _grid(rng, lo, hi):
    """Three grid counts with about lo..hi tets in all (log-uniform), none equal by construction."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi))) / 6
    e = cells ** (1 / 3)
    nx = max(3, round(e * rng.uniform(0.6, 1.5)))
    ny = max(2, round(math.sqrt(cells / nx) * rng.uniform(0.6, 1.2)))
    return dict(nx=nx, ny=ny, nz=max(3, round(cells / (nx * ny))))


def draw(rng) -> dict:
    kind = rng.choice(["assemble", "assemble", "drop_in", "apply", "apply", "sweep", "sweep", "lu", "direct",
                       "network"])
    c = dict(kind=kind)
    if kind == "assemble":
        c.update(family="guide", **_grid(rng, 1500, 340000), materials=rng.choice(["air", "lossy", "tensor"]))
    elif kind == "drop_in":
        c.update(family="guide", **_grid(rng, 1500, 24000), materials=rng.choice(["air", "lossy", "tensor"]))
    elif kind == "apply":
        nsys = rng.choice([1, 2, 3, 4, 5, 8, 13, 16, 27, 32, 40, 64])
        c.update(family="guide", **_grid(rng, 1500, min(75000, 1200000 // nsys)), materials=rng.choice(["air", "lossy"]),
                 nsys=nsys)
    elif kind == "sweep":
        pc, pr = rng.choice([("aux", "fp64"), ("aux", "mixed"), ("block_jacobi", "fp64")])
        hi = 1000 if pc == "block_jacobi" else 2500
        c.update(family="guide", **_grid(rng, 500, hi), materials="air", nfreq=rng.randint(1, 16),
                 nport=rng.choice([1, 2]), precond=pc, precision=pr)
    elif kind == "lu":
        n = rng.randint(5, 22)
        c.update(family="cavity", nx=n, ny=n, nz=n, materials="blocks", nrhs=rng.choice([1, 2, 3, 8, 11, 16]))
    elif kind == "direct":
        if rng.random() < 0.5:
            n = rng.randint(5, 15)
            c.update(family="cavity", nx=n, ny=n, nz=n, materials="blocks", nfreq=rng.randint(1, 9), nport=1,
                     precision="c64")
        else:
            c.update(family="substrate", nx=rng.randint(8, 12), ny=rng.randint(4, 8), nz=rng.randint(6, 9),
                     materials="layer", nfreq=rng.randint(1, 3), nport=2, precision="c128")
    else:
        c.update(family="guide", **_grid(rng, 1000, 6000), materials="air", nsys=rng.choice([1, 2, 3, 5, 8]))
    return c


# ----------------------------------------------------------------------------------------- inputs
def _problem(case, seed):
    fam, nx, ny, nz = case["family"], case["nx"], case["ny"], case["nz"]
    if fam == "cavity":
        return problems.cavity(n=nx, seed=seed)
    if fam == "substrate":
        return problems.substrate_box(nx, ny, nz, seed=seed, abc_order=1)
    P = problems.waveguide(nx=nx, ny=ny, nz=nz, seed=seed, shuffle_local=case["materials"] == "tensor")
    rng = np.random.default_rng(seed + 77)
    nt = P.mesh.n_tets
    if case["materials"] == "lossy":
        eps = rng.uniform(1, 10, nt) * (1 - 1j * rng.uniform(1e-4, 1e-2, nt))
        for i in range(3):
            P.er[i, i] = eps
    elif case["materials"] == "tensor":
        for t, scale in ((P.er, 4.0), (P.ur, 1.5)):
            t[:] = 0.1 * (rng.standard_normal(t.shape) + 1j * rng.standard_normal(t.shape))
            for i in range(3):
                t[i, i] += scale * (1 - 0.01j)
    return P


def _systems(case):
    nf = case.get("nfreq") or -(-case["nsys"] // 2)
    if case["family"] == "cavity":
        f = np.linspace(2e9, 6e9, 101)[46:46 + nf]            # neighbouring points of the 101-point sweep
    elif case["family"] == "substrate":
        f = np.linspace(1e9, 8e9, 51)[:nf]
    else:
        f = np.linspace(8e9, 12e9, nf) if nf > 1 else np.array([10e9])
    s = [(float(v), q) for v in f for q in range(case.get("nport", 2 if case["family"] != "cavity" else 1))]
    if case["kind"] == "apply":
        s = (s * case["nsys"])[:case["nsys"]]
    return s


def _rand(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    re = torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)
    return torch.complex(re, torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))


def _params(seed):
    """Network weights of the size that training works at (random output layer, so every layer counts)."""
    g = torch.Generator().manual_seed(seed)
    c = 32
    parts = [torch.randn(2 * c, generator=g) / c ** 0.5]
    for _ in range(8):
        parts.append(torch.eye(c).repeat(2, 1, 1).reshape(-1) * 0.5 + torch.randn(2 * c * c, generator=g) * 0.3 / c ** 0.5)
    parts.append(torch.randn(2 * c, generator=g) / c)
    return torch.cat(parts)


def _network_io(case, n_aux, seed):
    x = _rand((n_aux, case["nsys"]), seed + 5).to(torch.complex64)
    return x, _rand((n_aux, case["nsys"]), seed + 6).to(torch.complex64)


def prepare(case, seed):
    P = _problem(case, seed)
    kind = case["kind"]
    st = dict(kind=kind, case=case, P=P)
    if kind == "drop_in":
        return st
    if kind == "assemble":
        plan = CsrPlan(DeviceMesh(P.mesh, P.field))
        st.update(plan=plan, er=torch.from_numpy(P.er).cuda(), ur=torch.from_numpy(P.ur).cuda(),
                  E=torch.empty(plan.nnz, dtype=torch.complex128, device="cuda"),
                  B=torch.empty(plan.nnz, dtype=torch.complex128, device="cuda"))
        return st
    if kind == "network":
        aux = AuxSpace(P.mesh)
        x, dz = _network_io(case, aux.n_aux, seed)
        st.update(net=Network(aux, params=_params(seed)), x=x, dz=dz)
        return st
    sw = FrequencySweep(P)
    st.update(sw=sw, systems=_systems(case) if kind != "lu" else None)
    if kind == "apply":
        st["x"] = _rand((sw.n, case["nsys"]), seed + 3)
    elif kind == "lu":
        st.update(lu=sw.direct_solver(), f=float(P.freqs[50]), b=_rand((sw.n, case["nrhs"]), seed + 3))
        st["lu"].reserve(case["nrhs"])
    elif kind == "direct":
        sw.direct_solver().set_precision(case["precision"])
    elif case["precond"] == "aux":
        sw.aux_space().reserve(len(st["systems"]))
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "assemble":
        return list(st["plan"].assemble(st["er"], st["ur"], st["E"], st["B"]))
    if kind == "drop_in":
        E, B = tet_mass_stiffness_matrices(st["P"].field, st["P"].er, st["P"].ur)
        return [E.data, B.data, E.indices, E.indptr]
    if kind == "apply":
        return st["sw"].apply(st["systems"], st["x"])
    if kind == "sweep":
        return st["sw"].solve(st["systems"], tol=1e-8, maxit=40000, precond=case["precond"],
                              precision=case["precision"]).x
    if kind == "lu":
        return st["lu"].factor(st["f"]).solve(st["b"])
    if kind == "direct":
        return st["sw"].solve_direct(st["systems"], window=9, tol=1e-8, precision=case["precision"]).x
    za = st["net"].forward(st["x"])
    return [za, st["net"].backward(st["dz"])]


# ------------------------------------------------------------------------------------ work, tolerance
def _counts(case):
    """(tets, edges, faces, field DOFs, nonzeros of E) of the grid: nnz counts the ordered entity pairs
    that share a tet, by the simplex that the pair spans (1 per edge, 13 per face, 42 per tet), x 4."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nt = 6 * nx * ny * nz
    nf = (4 * nt + 4 * (nx * ny + ny * nz + nx * nz)) // 2
    ne = (nx + 1) * (ny + 1) * (nz + 1) + nf - nt - 1
    return nt, ne, nf, 2 * (ne + nf), 4 * (ne + 13 * nf + 42 * nt)


def work(case):
    nt, ne, nf, n, nnz = _counts(case)
    nn = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    mesh = 24 * nn + (4 + 6) * 8 * nt + 8 * ne + 18 * 16 * nt
    kind = case["kind"]
    if kind in ("assemble", "drop_in"):
        # inputs once, the values of E and B once (and the pattern where it is returned); the element sums:
        # 400 entries of two matrices, 4 complex multiply-adds by a real coefficient each
        return dict(bytes=mesh + 32 * nnz + (4 * (nnz + n) if kind == "drop_in" else 0), flops=400 * 2 * 4 * 4 * nt)
    if kind == "network":
        na = nn + ne
        rows = na * case["nsys"]
        # states are 32 complex64 per row and layer, forward once and backward twice (input and weights)
        return dict(bytes=8 * rows * 4 + 4 * 16512 * 2, flops=3 * 4 * 2 * rows * 2 * 2 * 32 * 32)
    nsys = case["nrhs"] if kind == "lu" else len(_systems(case))
    op = 36 * nnz + 4 * n
    vec = 2 * 16 * n * nsys
    if kind in ("apply", "sweep"):
        # a Krylov solve reads the operator at least once; its iterations depend on the method, not the path
        return dict(bytes=op + vec, flops=16 * nnz * nsys)
    # nested dissection of a cube: factor flops grow with the square of the tets and factor entries with
    # their power 4/3 (2.263e14 flops and 53 GB of complex64 factors at 384 000 tets)
    fl = 2.263e14 * (nt / 384000) ** 2
    fb = 53e9 * (nt / 384000) ** (4 / 3)
    return dict(bytes=op + vec + 2 * fb, flops=fl + fb * nsys)


def tolerance(case):
    """About four times the measured difference to ``exact`` where it has a value."""
    kind = case["kind"]
    if kind in ("assemble", "drop_in"):
        # 7e-14 at 384 000 tets: the cofactors of a small tet cancel in coordinates of the whole box
        return {"rel": 3e-13}
    if kind == "apply":
        return {"rel": 1e-13}
    if kind == "network":
        return {"rel": 2e-6}
    if kind == "lu":
        return {"rel": 1e-3}           # complex64 factors of an ill-conditioned system
    return {"rel": 2e-7}               # residual 1e-8 times the conditioning


# ------------------------------------------------------------------------------------------ exact
_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
_FACES = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]


def _vol(*v):
    """Integral of the product of barycentric coordinates over a tet of volume 1/6."""
    k = math.prod(math.factorial(v.count(i)) for i in range(4))
    return k / math.factorial(len(v) + 3)


def _mesh_tensors(P, dev):
    m = P.mesh
    nn = m.nodes.shape[1]
    nodes = torch.from_numpy(m.nodes).to(dev)
    v = torch.sort(torch.from_numpy(m.tets).to(dev), dim=0).values
    edges, tris = torch.from_numpy(m.edges).to(dev), torch.from_numpy(m.tris).to(dev)
    ek = edges[0] * nn + edges[1]
    fk = (tris[0] * nn + tris[1]) * nn + tris[2]
    ent = [torch.searchsorted(ek, v[a] * nn + v[b]) for a, b in _EDGES]
    ent += [torch.searchsorted(fk, (v[a] * nn + v[b]) * nn + v[c]) + m.n_edges for a, b, c in _FACES]
    return nodes, v, torch.stack(ent), m.n_edges + m.n_tris


def _elements(P, dev):
    """(dofs (20, nt), stiffness (nt, 20, 20), mass (nt, 20, 20)): each tet's vertices in ascending global
    order, so every entity is oriented alike; local DOFs are 6 edges, 4 faces (first kind), then the second."""
    nodes, v, ent, H = _mesh_tensors(P, dev)
    nt = v.shape[1]
    er = torch.from_numpy(P.er).to(dev).permute(2, 0, 1)
    iu = torch.linalg.inv(torch.from_numpy(P.ur).to(dev).permute(2, 0, 1))
    X = nodes[:, v].permute(2, 1, 0)                                        # (nt, vertex, xyz)
    J = X[:, 1:] - X[:, :1]
    V6 = torch.linalg.det(J).abs()
    g = torch.linalg.inv(J).transpose(1, 2)                                 # gradients of L1..L3
    g = torch.cat([-g.sum(1, keepdim=True), g], 1).to(torch.complex128)
    p = torch.einsum("tai,tij,tbj->tab", g, er, g) * V6[:, None, None]
    cr = torch.stack([torch.linalg.cross(g[:, a], g[:, b]) for a, b in _EDGES], 1)
    q = torch.einsum("tai,tij,tbj->tab", cr, iu, cr) * V6[:, None, None]
    ln = {}
    for a, b in _EDGES:
        ln[a, b] = ln[b, a] = (X[:, a] - X[:, b]).norm(dim=1)
    Q = lambda a, b, c, d: q[:, _EDGES.index((a, b)), _EDGES.index((c, d))]
    M = lambda a, b: p[:, a, b]
    D = torch.zeros((nt, 20, 20), dtype=torch.complex128, device=dev)
    F = torch.zeros_like(D)
    for i, (a, b) in enumerate(_EDGES):
        for j, (c, d) in enumerate(_EDGES):
            L = ln[a, b] * ln[c, d]
            for ki, x in ((0, a), (10, b)):
                for kj, y in ((0, c), (10, d)):
                    D[:, i + ki, j + kj] = 9 * L * Q(a, b, c, d) * _vol(x, y)
                    F[:, i + ki, j + kj] = L * (_vol(x, b, y, d) * M(a, c) - _vol(x, b, y, c) * M(a, d)
                                                - _vol(x, a, y, d) * M(b, c) + _vol(x, a, y, c) * M(b, d))
        for j, (c, d, f) in enumerate(_FACES):
            l1, l2 = ln[a, b] * ln[c, f], ln[a, b] * ln[c, d]
            qcf, qdf, qcd = Q(a, b, c, f), Q(a, b, d, f), Q(a, b, c, d)
            for ki, x in ((0, a), (10, b)):
                e1 = l1 * (-6 * _vol(x, d) * qcf - 3 * _vol(x, c) * qdf - 3 * _vol(x, f) * qcd)
                e2 = l2 * (6 * _vol(x, f) * qcd + 3 * _vol(x, d) * qcf - 3 * _vol(x, c) * qdf)
                m1 = l1 * (_vol(x, b, c, d) * M(a, f) - _vol(x, b, d, f) * M(a, c)
                           - _vol(x, a, c, d) * M(b, f) + _vol(x, a, d, f) * M(b, c))
                m2 = l2 * (_vol(x, b, d, f) * M(a, c) - _vol(x, b, f, c) * M(a, d)
                           - _vol(x, a, d, f) * M(b, c) + _vol(x, a, c, f) * M(b, d))
                for kj, e, mm in ((6, e1, m1), (16, e2, m2)):
                    D[:, i + ki, j + kj] = e
                    D[:, j + kj, i + ki] = e
                    F[:, i + ki, j + kj] = mm
                    F[:, j + kj, i + ki] = mm
    for i, (a, b, e) in enumerate(_FACES):
        for j, (c, d, f) in enumerate(_FACES):
            def curl(r, s, u):           # curl of L_r W_su against the column's first and second function
                cf, df, cd = Q(s, u, c, f), Q(s, u, d, f), Q(s, u, c, d)
                return (2 * _vol(r, d) * cf + _vol(r, c) * df + _vol(r, f) * cd,
                        -2 * _vol(r, f) * cd - _vol(r, d) * cf + _vol(r, c) * df)
            b_ae, a_be, e_ab = curl(b, a, e), curl(a, b, e), curl(e, a, b)
            lac, lab, lcf, lcd = ln[a, e], ln[a, b], ln[c, f], ln[c, d]
            for kj, n2, l2 in ((6, 0, lcf), (16, 1, lcd)):
                D[:, i + 6, j + kj] = lac * l2 * (2 * b_ae[n2] + a_be[n2] + e_ab[n2])
                D[:, i + 16, j + kj] = lab * l2 * (-2 * e_ab[n2] - b_ae[n2] + a_be[n2])
            # the mass block with the framework's index sets (it is not symmetric)
            F[:, i + 6, j + 6] = lac * lcf * (_vol(a, b, c, d) * M(e, f) - _vol(a, b, d, f) * M(e, c)
                                              - _vol(b, c, d, f) * M(a, f) + _vol(b, e, d, f) * M(a, c))
            F[:, i + 6, j + 16] = lac * lcd * (_vol(a, b, d, f) * M(e, c) - _vol(a, b, f, c) * M(e, d)
                                               - _vol(b, e, d, f) * M(a, c) + _vol(b, e, f, c) * M(a, d))
            F[:, i + 16, j + 6] = lab * lcf * (_vol(b, c, d, f) * M(a, f) - _vol(b, e, d, f) * M(a, c)
                                               - _vol(e, a, c, d) * M(b, f) + _vol(e, a, d, f) * M(b, c))
            F[:, i + 16, j + 16] = lab * lcd * (_vol(b, e, d, f) * M(a, c) - _vol(b, e, f, c) * M(a, d)
                                                - _vol(e, a, d, f) * M(b, c) + _vol(a, c, e, f) * M(b, d))
    return torch.cat([ent, ent + H]), D, F


_RULE = [(0.223381589678011, 0.108103018168070, 0.445948490915965), (0.109951743655322, 0.816847572980459,
                                                                     0.091576213509771)]


def _boundary(P, tri, shape, dev):
    """Robin blocks (ns, 8, 8) with coefficient 1, load vectors (ns, 8) of the field ``shape`` (3, points) and
    the DOFs (ns, 8) of the listed triangles: tangential basis functions at the degree-4, 6-point rule."""
    m = P.mesh
    t = torch.from_numpy(np.asarray(tri, dtype=np.int64)).to(dev)
    tn = torch.from_numpy(m.tris).to(dev)[:, t]
    X = torch.from_numpy(m.nodes).to(dev)[:, tn].permute(2, 1, 0)          # (ns, vertex, xyz)
    e1, e2 = X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]
    nrm = torch.linalg.cross(e1, e2)
    A2 = nrm.norm(dim=1)
    nh = nrm / A2[:, None]
    g = [torch.linalg.cross(nh, X[:, (i + 2) % 3] - X[:, (i + 1) % 3]) / A2[:, None] for i in range(3)]
    ln = lambda i, j: (X[:, i] - X[:, j]).norm(dim=1)
    R = torch.zeros((len(t), 8, 8), dtype=torch.float64, device=dev)
    b = torch.zeros((len(t), 8), dtype=torch.complex128, device=dev)
    for w, u, v in _RULE:
        for k in range(3):
            lam = [v, v, v]
            lam[k] = u
            W = lambda i, j: lam[i] * g[j] - lam[j] * g[i]
            N = [ln(i, j)[:, None] * lam[s] * W(i, j) for s_ in (0, 1) for i, j in ((0, 1), (1, 2), (0, 2))
                 for s in ((i, j)[s_],)]
            N = N[:3] + [-ln(0, 2)[:, None] * lam[1] * W(0, 2)] + N[3:] + [ln(0, 1)[:, None] * lam[2] * W(0, 1)]
            N = torch.stack(N, 1)                                            # (ns, 8, xyz)
            R += w * A2[:, None, None] / 2 * (N @ N.transpose(1, 2))
            if shape is not None:
                x = sum(lam[i] * X[:, i] for i in range(3))
                b += w * A2[:, None] / 2 * (N.to(torch.complex128) @ shape(x)[:, :, None])[..., 0]
    H = m.n_edges + m.n_tris
    te = torch.from_numpy(m.tri_to_edge).to(dev)[:, t].T
    dof = torch.cat([te, t[:, None] + m.n_edges, te + H, t[:, None] + m.n_edges + H], 1)
    return R.to(torch.complex128), b, dof


def _terms(P, case, dev):
    """Boundary terms [(coefficient(k0), blocks, dofs)] and per port (scale(k0), load, dofs)."""
    terms, loads = [], []
    for port in P.ports:
        if case["family"] == "substrate":
            d = torch.tensor([0.0, 0.0, 1.0], dtype=torch.complex128, device=dev)
            zs = 50.0 * port.width / port.height
            R, b, dof = _boundary(P, port.tri_ids, lambda x: d.expand(x.shape[0], 3), dev)
            terms.append((lambda k0, zs=zs: 1j * k0 * Z0 / zs, R, dof))
            loads.append((lambda k0, zs=zs, p=port: -2j * k0 * 10.0 / p.height * Z0 / zs, b, dof))
            continue
        w, h = port.dims
        ox = w / 2
        def shape(x, w=w, ox=ox):
            f = torch.cos(math.pi * (x[:, 0] - ox) / w).to(torch.complex128)
            return torch.stack([0 * f, f, 0 * f], 1)
        R, b, dof = _boundary(P, port.tri_ids, shape, dev)
        beta = lambda k0, w=w: math.sqrt(k0 ** 2 - (math.pi / w) ** 2)
        amp = math.sqrt(4 * Z0 / (w * h))
        mu0 = 1.0 / (C0 * C0 * 8.854187818814e-12)
        terms.append((lambda k0, beta=beta: 1j * beta(k0), R, dof))
        loads.append((lambda k0, beta=beta, amp=amp: -2j * beta(k0) * amp * math.sqrt(k0 * C0 * mu0 / beta(k0) / Z0), b, dof))
    for bc in P.robin:
        R, _, dof = _boundary(P, bc.tri_ids, None, dev)
        terms.append((lambda k0: 1j * k0, R, dof))
    return terms, loads


def _free(P, dev):
    m = P.mesh
    H = m.n_edges + m.n_tris
    t = torch.from_numpy(np.asarray(P.pec_tris, dtype=np.int64)).to(dev)
    e = torch.from_numpy(m.tri_to_edge).to(dev)[:, t].reshape(-1)
    free = torch.ones(2 * H, dtype=torch.bool, device=dev)
    for ids in (e, e + H, t + m.n_edges, t + m.n_edges + H):
        free[ids] = False
    return free


def _exact_csr(P, dev):
    dof, D, F = _elements(P, dev)
    n = 2 * (P.mesh.n_edges + P.mesh.n_tris)
    key = (dof.T[:, :, None] * n + dof.T[:, None, :]).reshape(-1)
    key, inv = torch.unique(key, return_inverse=True)
    out = [torch.zeros((len(key), 2), dtype=torch.float64, device=dev).index_add_(
        0, inv, torch.view_as_real(A.reshape(-1))) for A in (D, F)]
    rows = torch.bincount(key // n, minlength=n)
    ptr = torch.cat([torch.zeros(1, dtype=torch.int64, device=dev), torch.cumsum(rows, 0)])
    return [torch.view_as_complex(o) for o in out], (key % n).to(torch.int32), ptr.to(torch.int32)


def _exact_apply(P, case, x, dev):
    dof, D, F = _elements(P, dev)
    terms, _ = _terms(P, case, dev)
    free = _free(P, dev)
    y = torch.zeros_like(x)
    for s, (f, _) in enumerate(_systems(case)):
        k0 = 2 * math.pi * f / C0
        xs = x[:, s]
        acc = torch.zeros((x.shape[0], 2), dtype=torch.float64, device=dev)
        loc = torch.einsum("tij,jt->ti", D, xs[dof]) - k0 ** 2 * torch.einsum("tij,jt->ti", F, xs[dof])
        acc.index_add_(0, dof.T.reshape(-1), torch.view_as_real(loc.reshape(-1).contiguous()))
        for co, R, d in terms:
            v = co(k0) * (R @ xs[d][:, :, None])[..., 0]
            acc.index_add_(0, d.reshape(-1), torch.view_as_real(v.reshape(-1).contiguous()))
        y[:, s] = torch.view_as_complex(acc) * free
    return y


def _exact_solve(P, case, systems, b, dev):
    """Dense solves on the free DOFs; None where they would take too long."""
    free = _free(P, dev)
    nfree = int(free.sum())
    freqs = sorted({f for f, _ in systems})
    if 8 / 3 * nfree ** 3 * len(freqs) > 1e14 or nfree > 40000:
        return None
    dof, D, F = _elements(P, dev)
    terms, loads = _terms(P, case, dev)
    pos = torch.full((len(free),), nfree, dtype=torch.int64, device=dev)
    pos[free] = torch.arange(nfree, device=dev)
    out = torch.zeros((len(free), len(systems)), dtype=torch.complex128, device=dev)
    for f in freqs:
        k0 = 2 * math.pi * f / C0
        K = torch.zeros(((nfree + 1) ** 2, 2), dtype=torch.float64, device=dev)

        def add(d, v):
            i = pos[d]
            K.index_add_(0, (i[:, :, None] * (nfree + 1) + i[:, None, :]).reshape(-1),
                         torch.view_as_real(v.reshape(-1).contiguous()))
        add(dof.T, D - k0 ** 2 * F)
        for co, R, d in terms:
            add(d, co(k0) * R)
        A = torch.view_as_complex(K).reshape(nfree + 1, nfree + 1)[:nfree, :nfree].contiguous()
        del K
        cols = [j for j, (g, _) in enumerate(systems) if g == f]
        rhs = torch.zeros((len(free), len(cols)), dtype=torch.complex128, device=dev)
        for c, j in enumerate(cols):
            if b is not None:
                rhs[:, c] = b[:, j]
            else:
                sc, lv, d = loads[systems[j][1]]
                r = torch.view_as_real(rhs[:, c].contiguous())
                r.index_add_(0, d.reshape(-1), torch.view_as_real((sc(k0) * lv).reshape(-1).contiguous()))
                rhs[:, c] = torch.view_as_complex(r)
        x = torch.linalg.solve(A, rhs[free])
        for c, j in enumerate(cols):
            out[free, j] = x[:, c]
        del A
    return out


def _exact_network(P, case, seed, dev):
    m, C = P.mesh, 32
    nn, na = m.nodes.shape[1], m.nodes.shape[1] + m.n_edges
    x, dz = _network_io(case, na, seed)
    par = _params(seed).to(dev, torch.float64).requires_grad_(True)
    e = torch.from_numpy(m.edges).to(dev)
    eid = torch.arange(m.n_edges, device=dev) + nn
    src = torch.cat([eid, eid, e[0], e[1]])
    dst = torch.cat([e[0], e[1], eid, eid])
    deg = torch.bincount(dst, minlength=na).clamp(min=1).to(torch.float64)
    typ = (torch.arange(na, device=dev) >= nn).long()
    win, rest = par[:2 * C].reshape(2, C), par[2 * C:-2 * C].reshape(4, 2, 2, C, C)
    wout = par[-2 * C:].reshape(2, C)
    xr = torch.view_as_real(x.to(torch.complex128))                         # (na, S, 2)
    h = xr[:, :, :, None] * win[typ][:, None, None, :]
    for layer in range(4):
        msg = torch.zeros_like(h).index_add(0, dst, h[src]) / deg[:, None, None, None]
        W, U = rest[layer, 0], rest[layer, 1]
        h = torch.cat([h[:nn] @ W[0] + msg[:nn] @ U[0], h[nn:] @ W[1] + msg[nn:] @ U[1]])
    za = xr + (h * wout[typ][:, None, None, :]).sum(-1)
    (za * torch.view_as_real(dz.to(torch.complex128))).sum().backward()
    return [torch.view_as_complex(za.detach().contiguous()), par.grad]


def exact(case, seed):
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    P = _problem(case, seed)
    kind = case["kind"]
    if kind in ("assemble", "drop_in"):
        (E, B), idx, ptr = _exact_csr(P, dev)
        return [E, B] if kind == "assemble" else [E.cpu().numpy(), B.cpu().numpy(), None, None]
    if kind == "network":
        return _exact_network(P, case, seed, dev)
    n = 2 * (P.mesh.n_edges + P.mesh.n_tris)
    if kind == "apply":
        return _exact_apply(P, case, _rand((n, case["nsys"]), seed + 3), dev)
    if kind == "lu":
        f = float(P.freqs[50])
        return _exact_solve(P, case, [(f, j) for j in range(case["nrhs"])], _rand((n, case["nrhs"]), seed + 3), dev)
    return _exact_solve(P, case, _systems(case), None, dev)
