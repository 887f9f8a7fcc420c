"""Performance cases of the operator, its preconditioners and its solves, as a user's program calls
them: build a `DGOperator` on a mesh, set the material, autotune once, then apply / precondition /
solve on device vectors.

A case names one call: `task` is "apply" (y = A x), "bjacobi" (z = D^-1 r), "vcycle" (one multigrid
V-cycle) or "solve" (block-Jacobi CG from zero to `rtol`); `kind`, `dim`, `degree` the operator,
`mesh` with `n` the mesh ("box": the unit square or cube with curved boundary, "fault": the
antiplane domain graded toward a fault of `n` facets, "batch": a disjoint union of unit squares of
uneven sizes around n), `rule` the quadrature (tandem's tabulated rules, or the package's own
conical ones), `dtype` the vectors and arithmetic, `nrhs` the stacked right-hand sides.
"""
import json
import math
from math import comb
from pathlib import Path

import numpy as np
import torch

from tandem_b200 import mesh as M
from tandem_b200.operator import DGOperator, ELASTICITY, FP32, FP64, POISSON, Quadrature

ROOT = Path(__file__).resolve().parent.parent
KINDS = {"poisson": POISSON, "elasticity": ELASTICITY}
SMOOTH_ITS = 6  # Chebyshev steps per smoothing, as the benchmark's multigrid solves


def _case(name, task, kind, dim, degree, n, mesh="box", rule="tandem", dtype="f64", nrhs=1):
    return dict(name=name, task=task, kind=kind, dim=dim, degree=degree, mesh=mesh, n=n, rule=rule, dtype=dtype,
                nrhs=nrhs)


def listed():
    return [
        # the static elasticity solve's MatMult, 48,000 tetrahedra (5.04 M unknowns): the hot path
        _case("elasticity3d_p4", "apply", "elasticity", 3, 4, 20),
        # the same operator in FP32, as the reduced-precision solves run it (24,576 tetrahedra, the
        # inversion's mesh)
        _case("elasticity3d_p4_f32", "apply", "elasticity", 3, 4, 16, dtype="f32"),
        # a low-order run on a ragged mesh (7,986 tetrahedra: no multiple of a tile)
        _case("elasticity3d_p2", "apply", "elasticity", 3, 2, 11),
        # 3D Poisson with the package's own conical quadrature, odd size (13,182 tetrahedra)
        _case("poisson3d_p3", "apply", "poisson", 3, 3, 13, rule="conical"),
        # the 2D manufactured-solution test's MatMult (8,192 triangles): small, latency counts
        _case("poisson2d_p4", "apply", "poisson", 2, 4, 64),
        # a batch of Green's-function columns of the antiplane fault model in one call
        _case("poisson2d_p4_columns", "apply", "poisson", 2, 4, 96, mesh="fault", nrhs=32),
        # the uneven batch: independent 2D elasticity problems of different sizes as one operator
        _case("elasticity2d_p4_batch", "apply", "elasticity", 2, 4, 48, mesh="batch"),
        # the smallest call: a first-order operator on 162 triangles (a unit test, a coarse problem)
        _case("poisson2d_p1_small", "apply", "poisson", 2, 1, 9),
        # the default preconditioner of the static solve (10,368 tetrahedra, 105 x 105 blocks)
        _case("bjacobi_elasticity3d_p4", "bjacobi", "elasticity", 3, 4, 12),
        # the default preconditioner on Green's-function columns
        _case("bjacobi_poisson2d_p4_columns", "bjacobi", "poisson", 2, 4, 96, mesh="fault", nrhs=32),
        # the production preconditioner: one p-multigrid V-cycle (10,368 tetrahedra)
        _case("vcycle_elasticity3d_p4", "vcycle", "elasticity", 3, 4, 12),
        # a whole solve, tandem's default solver (block-Jacobi CG) on the 2D test problem
        _case("solve_poisson2d_p4", "solve", "poisson", 2, 4, 64),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    task = rng.choice(["apply"] * 7 + ["bjacobi"] * 2 + ["vcycle", "solve"])
    dim = 2 if task == "solve" else rng.choice([2, 3])
    degree = rng.choice([1, 2, 3, 4, 4, 4]) if task == "apply" else rng.choice([2, 3, 4])
    kind = "poisson" if task == "solve" else rng.choice(["poisson", "elasticity", "elasticity"])
    mesh = "box"
    if dim == 2 and task != "solve":
        mesh = rng.choice(["box", "batch"] + (["fault"] if kind == "poisson" else []))
    if dim == 3:
        n = log_int(2, 20 if task == "apply" else 12)
    else:
        n = {"fault": log_int(32, 128), "batch": log_int(4, 64)}.get(mesh) or log_int(4, 64 if task == "solve" else 128)
    case = dict(task=task, kind=kind, dim=dim, degree=degree, mesh=mesh, n=n,
                rule=rng.choice(["tandem", "tandem", "conical"]),
                dtype=rng.choice(["f64", "f64", "f32"]) if task in ("apply", "bjacobi") else "f64", nrhs=1)
    if dim == 2 and task != "solve" and rng.random() < 0.5:  # the largest listed call has 5.04 M unknowns
        case["nrhs"] = max(1, min(log_int(2, 48), int(5.0e6 / (_elements(case) * _bs(case)))))
    return case


# ---- sizes --------------------------------------------------------------------------------------


def _components(case):
    return 1 if case["kind"] == "poisson" else case["dim"]


def _bs(case):
    return comb(case["degree"] + case["dim"], case["dim"]) * _components(case)


def _batch_cells(n):
    """Cells per direction of the batch's problems: uneven around n (element counts spread 1 : 16)."""
    return [max(2, int(round(n * s))) for s in (0.5, 1.0, 0.35, 0.8, 1.4, 0.6)]


def _elements(case):
    if case["mesh"] == "batch":
        return sum(2 * c * c for c in _batch_cells(case["n"]))
    if case["mesh"] == "fault":
        return 2 * (_fault_mesh(case).info["nx"] - 1) * (_fault_mesh(case).info["ns"] - 1)
    return (2 if case["dim"] == 2 else 6) * case["n"] ** case["dim"]


def _facets(case):
    """Facets, and those of them on the boundary (box-like meshes)."""
    if case["mesh"] == "batch":
        per = [(3 * c * c + 2 * c, 4 * c) for c in _batch_cells(case["n"])]
        return sum(a for a, _ in per), sum(b for _, b in per)
    if case["mesh"] == "fault":
        m = _fault_mesh(case)
        x, s = m.info["nx"] - 1, m.info["ns"] - 1
        return 3 * x * s + x + s, 2 * (x + s)
    n = case["n"]
    return (3 * n * n + 2 * n, 4 * n) if case["dim"] == 2 else (12 * n ** 3 + 6 * n * n, 12 * n * n)


def work(case):
    D, Q, N, bs, E = case["dim"], _components(case), case["degree"], _bs(case), _elements(case)
    F, FB = _facets(case)
    q = _quadrature(case)
    Nq, nq, nbf, s, r = len(q.vol_w), len(q.fct_w), bs // Q, 4 if case["dtype"] == "f32" else 8, case["nrhs"]
    ncoef = 1 if Q == 1 else 2
    # one operator apply: every geometry and coefficient value once, the vectors once per column;
    # every facet flux once for both sides
    geo = (E * (D * D + ncoef) * Nq + F * (D + 1 + 2 * D * D + (0 if Q == 1 else 4)) * nq) * s
    vec = 2 * E * bs * s
    vol = 4 * nbf * D * Nq * Q + (4 * D * D * Q + 3 * D * D) * Nq
    fct = 8 * nbf * (D + 1) * Q * nq + (8 * D * D * Q + 18 * D * D) * nq
    flops = E * vol + (F - FB / 2) * fct
    # block-Jacobi: the symmetric inverses once, the vectors once per column
    jac = dict(bytes=E * bs * (bs + 1) / 2 * s + r * vec, flops=2 * E * bs * bs * r)
    if case["task"] == "apply":
        return dict(bytes=geo + r * vec, flops=r * flops)
    if case["task"] == "bjacobi":
        return jac
    if case["task"] == "solve":  # about 34 n iterations at degree 4, fewer below
        its = max(8, int(34 * case["n"] * N * N / 16))
        return dict(bytes=its * (geo + vec + jac["bytes"] + 6 * vec), flops=its * (flops + jac["flops"]))
    # the V-cycle: 2 x steps applies on the finest level and on the block-sparse levels below it
    fine = 2 * SMOOTH_ITS
    levels, d = 0, N
    while d > 1:
        d = max(1, d // 2)
        levels += (D + 2) * (comb(d + D, D) * Q) ** 2
    return dict(bytes=fine * (geo + r * vec + E * levels * s), flops=r * fine * (flops + 2 * E * levels))


# ---- inputs -------------------------------------------------------------------------------------


def _quadrature(case):
    """The rules of order 2 N + 1: tandem's own (the repository's fixture), or the package's conical ones."""
    order, D = 2 * case["degree"] + 1, case["dim"]
    if case["rule"] == "conical":
        return Quadrature.conical(D, order)
    rules = json.loads((ROOT / "tests" / "golden" / "quadrature.json").read_text())["auto"]
    v, f = rules[f"{D}:{order}"], rules[f"{D - 1}:{order}"]
    return Quadrature(np.array(v["points"]).reshape(-1, D), np.array(v["weights"]),
                      np.array(f["points"]).reshape(-1, D - 1), np.array(f["weights"]))


def _fault_mesh(case):
    return M.graded_fault_mesh(case["n"])


def _mesh(case):
    N = case["degree"]
    if case["mesh"] == "fault":
        m = _fault_mesh(case)
        M.topology(m, m.info["boundary_bc"], m.info["interior_bc"])
        return M.geometry_nodes(m, N)
    curve = M.box_boundary_surface(0.02)
    if case["mesh"] == "batch":
        return M.union([M.build(M.square_mesh(c), N, curve=curve) for c in _batch_cells(case["n"])])[0]
    return M.build(M.square_mesh(case["n"]) if case["dim"] == 2 else M.cube_mesh(case["n"]), N, curve=curve)


def _field(X, rng):
    """A smooth positive random field at the points X [..., D] (log of a few random waves)."""
    k = rng.normal(size=(4, X.shape[-1])) * 2.5
    s = sum(np.sin(X @ k[i] + p) for i, p in enumerate(rng.uniform(0, 2 * np.pi, 4)))
    return np.exp(0.25 * s)


def _material(case, X, seed):
    rng = np.random.default_rng(1000 + seed)
    if case["mesh"] == "fault":  # a homogeneous half space, its modulus from the seed
        return np.full(X.shape[:2], rng.uniform(0.5, 2.0)), None
    return _field(X, rng), (_field(X, rng) if case["kind"] == "elasticity" else None)


def _vector(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    return torch.randn(case["nrhs"], _elements(case) * _bs(case), dtype=dt, device="cuda", generator=g)


def prepare(case, seed):
    m = _mesh(case)
    op = DGOperator(m, case["degree"], KINDS[case["kind"]], _quadrature(case))
    X = op.volume_coords()
    op.set_material(*_material(case, X, seed))
    prec = FP32 if case["dtype"] == "f32" else FP64
    state = dict(case=case, op=op, prec=prec, nrhs=case["nrhs"])
    if case["task"] != "bjacobi":
        op.autotune(prec, nrhs=case["nrhs"])
    if case["task"] in ("bjacobi", "solve"):
        op.bjacobi_setup(prec)
    if case["task"] == "vcycle":
        op.mg_setup(smooth_its=SMOOTH_ITS)
    if case["task"] == "solve":  # a smooth load
        f = np.log(_field(X, np.random.default_rng(2000 + seed)))[:, None, :]
        state["x"] = torch.as_tensor(op.rhs(f), device="cuda")
    else:
        state["x"] = _vector(case, seed)
    state["y"] = torch.empty_like(state["x"])
    return state


def run(state):
    op, x, y = state["op"], state["x"], state["y"]
    task = state["case"]["task"]
    if task == "apply":
        op.apply(x, y, state["prec"], nrhs=state["nrhs"])
    elif task == "bjacobi":
        op.bjacobi_apply(x, y, state["prec"], nrhs=state["nrhs"])
    elif task == "vcycle":
        op.mg_apply(x, y, nrhs=state["nrhs"])
    else:
        y.zero_()
        op.solve(x, y, rtol=1e-10)
    return y


# ---- the same in plain FP64 torch ---------------------------------------------------------------


def _jacobi_hom(n, a, x, y):
    """y^n P_n^(a,0)(x / y) from the explicit sum."""
    return sum(comb(n + a, n - s) * comb(n, s) * ((x - y) / 2) ** s * ((x + y) / 2) ** (n - s) for s in range(n + 1))


def _modes(D, N):
    """Exponents of the modal basis: by total degree, the first component decreasing."""
    if D == 2:
        return [(d - j, j) for d in range(N + 1) for j in range(d + 1)]
    return [(i, j, d - i - j) for d in range(N + 1) for i in range(d, -1, -1) for j in range(d - i, -1, -1)]


def _dubiner(D, N, p):
    """The modal basis at points p [np, D] -> [np, Nbf]."""
    out = []
    for e in _modes(D, N):
        if D == 2:
            v = _jacobi_hom(e[0], 0, 2 * p[:, 0] - 1 + p[:, 1], 1 - p[:, 1])
            v = v * _jacobi_hom(e[1], 2 * e[0] + 1, 2 * p[:, 1] - 1, 1 + 0 * p[:, 1])
        else:
            v = _jacobi_hom(e[0], 0, 2 * p[:, 0] - 1 + p[:, 1] + p[:, 2], 1 - p[:, 1] - p[:, 2])
            v = v * _jacobi_hom(e[1], 2 * e[0] + 1, 2 * p[:, 1] - 1 + p[:, 2], 1 - p[:, 2])
            v = v * _jacobi_hom(e[2], 2 * e[0] + 2 * e[1] + 2, 2 * p[:, 2] - 1, 1 + 0 * p[:, 2])
        out.append(v)
    return np.stack(out, axis=1)


def _monomials(D, N, p):
    """Monomials at p [np, D] -> [np, Nbf] and their gradients [np, D, Nbf]."""
    ex = np.array(_modes(D, N))
    v = np.prod(p[:, None, :] ** ex[None], axis=2)
    g = np.stack([ex[:, d] * p[:, None, d] ** np.maximum(ex[:, d] - 1, 0) *
                  np.prod(np.delete(p[:, None, :] ** ex[None], d, axis=2), axis=2) for d in range(D)], axis=1)
    return v, g


def _nodes(D, N):
    """The basis nodes: a mesh's degree-N geometry nodes on the unit simplex."""
    ref = M.SimplexMesh(D, np.vstack([np.zeros(D), np.eye(D)]), np.arange(D + 1)[None])
    return M.geometry_nodes(ref, N).geo_nodes[0]


def _basis(D, N, nodal, p):
    """Values [np, Nbf] and gradients [np, D, Nbf] of the basis at p, as tensors on the GPU."""
    z = _nodes(D, N)
    v, g = _monomials(D, N, p)
    c = np.linalg.inv(_monomials(D, N, z)[0])  # monomial coefficients of the Lagrange basis
    if not nodal:
        c = c @ _dubiner(D, N, z)
    return torch.as_tensor(v @ c, device="cuda"), torch.as_tensor(g @ c, device="cuda")


def _exact_operator(case, seed):
    """f(U, own) = A U for U [E, Q, Nbf] in FP64; own=True: only the element's own diagonal block."""
    D, N, Q = case["dim"], case["degree"], _components(case)
    m, q = _mesh(case), _quadrature(case)

    def dev(a):
        return torch.as_tensor(np.ascontiguousarray(a), device="cuda")

    nodal = case["kind"] == "elasticity"
    X, W, w = dev(m.geo_nodes), dev(q.vol_w), dev(q.fct_w)

    def geometry(els, gd):
        """|det J| and J^-1 [.., q, a, i] of elements els from geometry gradients gd [q, a, n]."""
        J = torch.einsum("eni,qan->eqia", X[els], gd)
        return torch.linalg.det(J).abs(), torch.linalg.inv(J)

    every = torch.arange(m.num_elements, device="cuda")
    _, gD = _basis(D, m.geo_degree, True, q.vol_x)
    gE, _ = _basis(D, m.geo_degree, True, q.vol_x)
    det, G = geometry(every, gD)
    _, dV = _basis(D, N, nodal, q.vol_x)  # [q, a, k]
    pts = torch.einsum("eni,qn->eqi", X, gE).cpu().numpy()
    mats = [dev(c) for c in _material(case, pts, seed) if c is not None]
    mV, _ = _basis(D, N, True, q.vol_x)
    mass = torch.einsum("qk,eq,ql->ekl", mV, W * det, mV)
    nod = [torch.linalg.solve(mass, torch.einsum("eq,qk->ek", c * W * det, mV)[..., None])[..., 0] for c in mats]
    coef = [(c @ mV.T) * W * det for c in nod]
    size = (W * det).sum(1)
    lo, hi = (nod[0], nod[0]) if Q == 1 else (2 * nod[1], D * nod[0] + 2 * nod[1])
    stiff = hi.amax(1) ** 2 / lo.amin(1)  # c1^2 / c0 of the penalty

    # facets by (local face of side 0, of side 1, boundary or not)
    verts = np.vstack([np.zeros(D), np.eye(D)])
    faces = [tuple(j for j in range(D + 1) if j != D - f) for f in range(D + 1)]  # D-subsets in order
    chi = q.fct_x
    tab = []
    for f in faces:
        p = (1 - chi.sum(1))[:, None] * verts[f[0]] + sum(chi[:, d:d + 1] * verts[f[d + 1]] for d in range(D - 1))
        missing = next(v for v in range(D + 1) if v not in f)
        nref = np.ones(D) if missing == 0 else -np.eye(D)[missing - 1]  # outward, scaled
        tab.append((_basis(D, N, nodal, p), _basis(D, m.geo_degree, True, p)[1], _basis(D, N, True, p)[0], dev(nref)))
    groups = []
    up, loc, bc = m.facet_up, m.facet_local, m.facet_bc
    bnd = up[:, 0] == up[:, 1]
    flux = np.where(bnd, (bc == M.BC_FAULT) | (bc == M.BC_DIRICHLET), bc != M.BC_NATURAL)
    assert not (bnd & (bc == M.BC_NONE)).any()
    cn = N * (N - 1 + D) / D
    for b in (False, True):
        for l0 in range(D + 1):
            for l1 in range(D + 1):
                ids = np.nonzero(flux & (bnd == b) & (loc[:, 0] == l0) & (loc[:, 1] == l1))[0]
                if not len(ids):
                    continue
                e = [dev(up[ids, s]) for s in (0, 1)]
                t = [tab[l0], tab[l1]]
                d0, G0 = geometry(e[0], t[0][1])
                G1 = geometry(e[1], t[1][1])[1]
                n = d0[..., None] * torch.einsum("fqai,a->fqi", G0, t[0][3])
                nl = n.norm(dim=2)
                area = (w * nl).sum(1)
                p = [(D + 1) * cn * area / size[x] * stiff[x] for x in e]
                pen = p[0] if b else (p[0] + p[1]) / 4
                mt = [[c[e[s]] @ t[s][2].T for c in nod] for s in (0, 1)]
                groups.append((b, e, t, n, pen[:, None] * nl, (G0, G1), mt))

    def stress(cs, J):
        """The flux tensor [.., i, r] of physical gradients J [.., i, r] (i the derivative)."""
        if Q == 1:
            return cs[0][..., None, None] * J
        tr = J.diagonal(dim1=-2, dim2=-1).sum(-1)
        return cs[1][..., None, None] * (J + J.transpose(-1, -2)) + \
            (cs[0] * tr)[..., None, None] * torch.eye(D, dtype=J.dtype, device=J.device)

    def act(U, own=False):
        g = torch.einsum("erk,qak->eqar", U, dV)
        T = torch.einsum("eqai,eqir->eqar", G, stress(coef, torch.einsum("eqai,eqar->eqir", G, g)))
        Y = torch.einsum("eqar,qak->erk", T, dV)
        for b, e, t, n, pn, Gs, mt in groups:
            sides = (0,) if b else (0, 1)
            u = [torch.einsum("frk,qk->fqr", U[e[s]], t[s][0][0]) for s in sides]
            tr = [torch.einsum("fqi,fqir->fqr", n, stress(mt[s], torch.einsum(
                "fqai,fqar->fqir", Gs[s], torch.einsum("frk,qak->fqar", U[e[s]], t[s][0][1])))) for s in sides]
            for s in sides:
                sg = 1.0 if s == 0 else -1.0
                if b:
                    jump, avg = u[0], tr[0]
                    lift = -u[0]
                else:
                    o = 0.0 if own else 1.0  # the other side's part
                    us = [u[0], o * u[1]] if s == 0 else [o * u[0], u[1]]
                    ts = [tr[0], o * tr[1]] if s == 0 else [o * tr[0], tr[1]]
                    jump, avg, lift = us[0] - us[1], (ts[0] + ts[1]) / 2, (us[1] - us[0]) / 2
                val = -sg * (avg - pn[..., None] * jump)
                S = stress(mt[s], n[..., :, None] * lift[..., None, :])
                # the lift's stress is that of the symmetric pair: n (x) lift as a displacement gradient
                gr = torch.einsum("fqai,fqir->fqar", Gs[s], S)
                c = torch.einsum("q,fqr,qk->frk", w, val, t[s][0][0]) + torch.einsum("q,fqar,qak->frk", w, gr, t[s][0][1])
                Y.index_add_(0, e[s], c)
        return Y

    return act


def exact(case, seed):
    if case["task"] in ("vcycle", "solve"):
        return None  # an iteration's result, not a closed form
    E, Q = _elements(case), _components(case)
    nbf = _bs(case) // Q
    act = _exact_operator(case, seed)
    X = _vector(case, seed).double().reshape(case["nrhs"], E, Q, nbf)
    if case["task"] == "apply":
        Y = torch.stack([act(x) for x in X])
    else:
        cols = []
        for j in range(Q * nbf):
            U = torch.zeros(E, Q * nbf, dtype=torch.float64, device="cuda")
            U[:, j] = 1.0
            cols.append(act(U.reshape(E, Q, nbf), own=True).reshape(E, -1))
        A = torch.stack(cols, dim=2)
        Y = torch.linalg.solve(A, X.reshape(case["nrhs"], E, -1).permute(1, 2, 0)).permute(2, 0, 1)
    return Y.reshape(case["nrhs"], -1)
