"""The calls this library is used for, as timed cases.

Three kinds of work, each through the public classes:

  assemble        ``NavierStokes.assemble`` + ``apply_dirichlet``: one time step's linear system
                  (LinearizeU, element assembly into the CSR values, symmetric Dirichlet conditions);
                  ``members`` > 1 does it for a ``Batch`` of meshes in one call.
  step            ``NavierStokes.step``: whole coupled time steps (assembly, Krylov solve, update),
                  then the fields are read back; ``members`` > 1 steps a ``Batch``.
  semi            ``NavierStokesSemiImplicit.step``: predictor/corrector steps, then the fields are read.

Meshes are jittered structured triangulations and Kuhn tetrahedra, the assembly cases with the
conditions of a lid-driven cavity, the time steps with those of a channel (parabolic inlet, no-slip
walls, p = 0 at the outlet).  ``order`` = "random" numbers nodes and elements as an unstructured mesh
generator does.
"""
import itertools
import math

import numpy as np
import torch

from coolfluid3_b200 import Batch, NavierStokes, NavierStokesSemiImplicit


def _case(name, kind, dim, cells, **more):
    c = {"name": name, "kind": kind, "dim": dim, "cells": cells, "members": 1, "form": "generic",
         "order": "natural", "nu": 1e-2, "dt": 1e-2}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: 64 x 64 cells of triangles in the default (specialised) element form
        _case("tri_64_spec", "assemble", 2, 64, form="specialised"),
        # an odd-sized, unstructured triangle mesh in the generic form
        _case("tri_301_generic_random", "assemble", 2, 301, order="random"),
        # a small tetrahedron mesh as in interactive or served use
        _case("tet_17_spec", "assemble", 3, 17, form="specialised", nu=1e-3, dt=5e-3),
        # the benchmark's mesh: 64^3 x 6 tetrahedra, generic form
        _case("tet_64_generic", "assemble", 3, 64, nu=1e-3, dt=5e-3),
        # a mid-sized unstructured tetrahedron mesh, default form
        _case("tet_37_spec_random", "assemble", 3, 37, form="specialised", order="random", nu=1e-3, dt=5e-3),
        # the largest: 96^3 x 6 = 5.3 million tetrahedra, default form
        _case("tet_96_spec", "assemble", 3, 96, form="specialised", nu=1e-3, dt=5e-3),
        # many small meshes assembled in one call
        _case("batch_tri_assemble", "assemble", 2, 96, members=16),
        # coupled time steps of a 2D channel at the 64 x 64 configuration's size, point Jacobi
        _case("step_tri_64", "step", 2, 64, steps=2, precond="jacobi", precision="fp64"),
        # coupled time steps of a 3D channel with the two-level preconditioner
        _case("step_tet_24_two_level", "step", 3, 24, steps=2, precond="two_level_coupled", precision="fp64",
              nu=1e-2, dt=1e-2),
        # FP32 element matrices refined to the FP64 answer, 623,000 tetrahedra
        _case("step_tet_47_mixed", "step", 3, 47, steps=2, precond="two_level_coupled", precision="fp32",
              nu=1e-2, dt=1e-2),
        # a batch of small 2D channels stepped together
        _case("batch_step_tri_40", "step", 2, 40, members=8, steps=1, precond="jacobi", precision="fp64"),
        # semi-implicit steps in 3D
        _case("semi_tet_32", "semi", 3, 32, steps=2),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    dim = rng.choice([2, 3])
    nu = 10.0 ** rng.uniform(-3.0, -1.5)
    dt = 10.0 ** rng.uniform(-2.3, -2.0)
    r = rng.random()
    if r < 0.55:
        members = rng.choice([1, 1, 1, 6, 11])
        hi = (400 if dim == 2 else 80) if members == 1 else (120 if dim == 2 else 20)
        return {"kind": "assemble", "dim": dim, "cells": size(9 if dim == 3 else 40, hi), "members": members,
                "form": rng.choice(["generic", "specialised"]), "order": rng.choice(["natural", "random"]),
                "nu": nu, "dt": dt}
    if r < 0.8:
        members = rng.choice([1, 1, 5])
        hi = 72 if dim == 2 else 36
        if members > 1:
            hi = 40 if dim == 2 else 12
        return {"kind": "step", "dim": dim, "cells": size(8 if dim == 3 else 20, hi), "members": members,
                "form": rng.choice(["generic", "specialised"]), "order": rng.choice(["natural", "random"]),
                "nu": nu, "dt": dt, "steps": rng.choice([1, 2]),
                "precond": rng.choice(["jacobi", "two_level_coupled"]), "precision": rng.choice(["fp64", "fp32"])}
    return {"kind": "semi", "dim": dim, "cells": size(8 if dim == 3 else 20, 100 if dim == 2 else 30), "members": 1,
            "form": "generic", "order": rng.choice(["natural", "random"]), "nu": nu, "dt": dt,
            "steps": rng.choice([1, 2])}


# ---- meshes, fields and conditions ------------------------------------------------


def _mesh(dim, n, seed, order, jitter=0.15):
    """(coords, conn, ijk) of n cells a side (n + 1 of them in the last direction of odd 2D sizes)."""
    rng = np.random.default_rng(seed)
    s = n + 1
    ax = np.arange(s)
    ijk = np.stack([g.ravel() for g in np.meshgrid(*([ax] * dim), indexing="ij")][::-1], axis=1)  # x fastest
    coords = ijk / float(n)
    interior = np.all((ijk > 0) & (ijk < n), axis=1)
    coords[interior] += rng.uniform(-jitter / n, jitter / n, (int(interior.sum()), dim))
    stride = s ** np.arange(dim)
    cell = np.stack([g.ravel() for g in np.meshgrid(*([np.arange(n)] * dim), indexing="ij")][::-1], axis=1) @ stride
    conn = []
    for perm in itertools.permutations(range(dim)):  # the Kuhn split of the cell
        v = np.cumsum([0] + [int(stride[p]) for p in perm])
        if _odd(perm):
            v[[0, 1]] = v[[1, 0]]  # positive orientation
        conn.append(cell[:, None] + v[None, :])
    conn = np.stack(conn, axis=1).reshape(-1, dim + 1)
    if order == "random":
        new = rng.permutation(len(coords))  # node i becomes node new[i]
        old = np.argsort(new)
        coords, ijk, conn = coords[old], ijk[old], new[conn]
        conn = conn[rng.permutation(len(conn))]
    return np.ascontiguousarray(coords), np.ascontiguousarray(conn.astype(np.uint32)), ijk


def _odd(perm):
    return sum(perm[i] > perm[j] for i in range(len(perm)) for j in range(i + 1, len(perm))) % 2 == 1


def _inlet(c, dim):
    u = 4.0 * c[:, 1] * (1.0 - c[:, 1])
    return u if dim == 2 else u * 4.0 * c[:, 2] * (1.0 - c[:, 2])


def _problem(case, seed, member=0):
    dim, n = case["dim"], case["cells"]
    if case["members"] > 1:  # members of different sizes
        n = max(4, n - (5 * member) % max(1, n // 2))
    coords, conn, ijk = _mesh(dim, n, 1000 * seed + member, case["order"])
    rng = np.random.default_rng(1000 * seed + 500 + member)
    N = len(coords)

    def modes(amplitude):
        u = np.zeros((N, dim))
        for c in range(dim):
            for _ in range(3):
                k, ph = rng.integers(1, 4, dim), rng.uniform(0.0, 2.0 * math.pi, dim)
                u[:, c] += amplitude / 3.0 * np.prod(np.sin(math.pi * k * coords + ph), axis=1)
        return u

    if case["kind"] == "assemble":  # lid-driven cavity in the middle of a run: a history that differs
        u = modes(1.0)
        hist = [u - 0.02 * (k + 1) * modes(1.0) for k in range(3)]
        up = np.concatenate([u, 0.1 * modes(1.0)[:, :1]], axis=1)
        lin = np.concatenate([u] + hist, axis=1)
        nodes, comps, vals = [], [], []
        for axis in range(dim):
            for side in (0, n):
                ids = np.nonzero(ijk[:, axis] == side)[0]
                lid = axis == dim - 1 and side == n
                nodes.append(np.repeat(ids, dim))
                comps.append(np.tile(np.arange(dim), len(ids)))
                vals.append(np.where(np.tile(np.arange(dim), len(ids)) == 0, 1.0 if lid else 0.0, 0.0))
        nodes.append(np.array([0]))
        comps.append(np.array([dim]))
        vals.append(np.array([0.0]))
    else:  # channel along x
        bump = np.prod(np.sin(math.pi * coords), axis=1)[:, None]
        u = 0.2 * bump * modes(1.0)
        u[:, 0] += _inlet(coords, dim)
        up = np.concatenate([u, np.zeros((N, 1))], axis=1)
        lin = np.tile(u, (1, 4))
        wall = np.any((ijk[:, 1:] == 0) | (ijk[:, 1:] == n), axis=1)
        inlet = np.nonzero((ijk[:, 0] == 0) & ~wall)[0]
        walls, out = np.nonzero(wall)[0], np.nonzero((ijk[:, 0] == n) & ~wall)[0]
        nodes, comps, vals = [], [], []
        for ids, values in ((walls, np.zeros(len(walls))), (inlet, _inlet(coords[inlet], dim))):
            for c in range(dim):
                nodes.append(ids)
                comps.append(np.full(len(ids), c))
                vals.append(values if c == 0 else np.zeros(len(ids)))
        nodes.append(out)
        comps.append(np.full(len(out), dim))
        vals.append(np.zeros(len(out)))
    bc = (np.concatenate(nodes).astype(np.uint32), np.concatenate(comps).astype(np.int32), np.concatenate(vals))
    nu = case["nu"] * (1.0 + 0.2 * np.cos(math.pi * coords[:, 0]))
    return {"coords": coords, "conn": conn, "up": up, "lin": np.ascontiguousarray(lin), "nu": nu, "bc": bc}


# ---- the measured calls -----------------------------------------------------------


class _View:
    """A device array of the library, seen by torch without a copy; keeps the handle that owns it."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (int(ptr), False), "version": 3}


def _view(owner, ptr, n):
    return torch.as_tensor(_View(owner, ptr, n), device="cuda")


def _solver(case, pb):
    ns = NavierStokes(pb["coords"], pb["conn"], dt=case["dt"], use_specializations=case["form"] == "specialised",
                      precision=case.get("precision", "fp64"))
    ns.set_state(pb["up"], pb["lin"], pb["nu"])
    ns.add_dirichlet(*pb["bc"])
    return ns


def _krylov(case):
    mixed = "matrix_free" if case["precision"] == "fp32" else False
    return {"method": "bicgstab", "precond": case["precond"], "tol": 1e-12, "max_iters": 4000, "mixed": mixed}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "semi":
        pb = _problem(case, seed)
        dim = case["dim"]
        si = NavierStokesSemiImplicit(pb["coords"], pb["conn"], dt=case["dt"], theta=0.5)
        si.set_krylov(velocity={"tol": 1e-12}, pressure={"tol": 1e-12})
        si.initial_conditions(pb["up"][:, :dim], pb["nu"])
        nodes, comps, vals = pb["bc"]
        for c in range(dim):
            si.add_velocity_dirichlet(nodes[comps == c], c, vals[comps == c])
        si.add_pressure_dirichlet(nodes[comps == dim], vals[comps == dim])
        return {"case": case, "solver": si}
    members = [_solver(case, _problem(case, seed, m)) for m in range(case["members"])]
    state = {"case": case, "solver": members[0], "members": members}
    if case["members"] > 1:
        state["batch"] = Batch(members)
    if kind == "assemble":
        state["out"] = []
        for m in members:
            v = m.device_view()
            state["out"].append({"values": _view(m, v["vals"], v["nnz"]), "rhs": _view(m, v["rhs"], v["nb_rows"])})
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "semi":
        si = state["solver"]
        si.step(case["steps"])
        return dict(zip(("solution", "linearized"), si.state))
    batch = state.get("batch")
    if case["kind"] == "assemble":
        if batch is not None:
            batch.assemble()
        else:
            state["solver"].assemble()
            state["solver"].apply_dirichlet()
        return state["out"]
    if batch is not None:
        for _ in range(case["steps"]):
            batch.step(**_krylov(case))
    else:
        state["solver"].step(case["steps"], **_krylov(case))
    return [dict(zip(("solution", "linearized"), m.state())) for m in state["members"]]


# ---- what a pass cannot do without ------------------------------------------------


def _counts(case, member):
    dim, n = case["dim"], case["cells"]
    if case["members"] > 1:
        n = max(4, n - (5 * member) % max(1, n // 2))
    N, E = (n + 1) ** dim, math.factorial(dim) * n ** dim
    edges = 3 * n * n + 2 * n if dim == 2 else 7 * n ** 3 + 9 * n * n + 3 * n
    return N, E, N + 2 * edges


def work(case):
    """Bytes: connectivity, node fields and coordinates read, CSR values and RHS written (assembly); for a
    solve, one read of the matrix and the vectors per product, two products (one for CG) an iteration, with
    an iteration count that grows with the cells a side.  Flops likewise."""
    dim = case["dim"]
    b = f = 0.0
    for m in range(case["members"]):
        N, E, nb = _counts(case, m)
        neq = dim + 1
        fields = N * 8.0 * (dim + 4 * dim + neq + 1)
        asm = E * (dim + 1) * 4.0 + fields + nb * neq * neq * 8.0 + N * neq * 8.0
        asm_f = E * (1650.0 if dim == 3 else 450.0)
        if case["kind"] == "assemble":
            b, f = b + asm, f + asm_f
            continue
        it = (1.0 if case["kind"] == "semi" or case["precond"] != "jacobi" else 2.5) * case["cells"] + 20.0
        if case["kind"] == "semi":
            mat = nb * (dim * dim + 1) * 8.0
            solve, solve_f = 2 * it * mat, 4 * it * nb * (dim * dim + 1)
            asm = asm * 0.6
        else:
            mat = nb * neq * neq * (8.0 if case["precision"] == "fp64" else 4.0)
            solve, solve_f = 2 * it * mat, 4 * it * nb * neq * neq
        b += case["steps"] * (asm + solve + 2 * fields)
        f += case["steps"] * (asm_f + solve_f)
    return {"bytes": b, "flops": f}


# ---- the same outputs in 64 bits by plain torch -------------------------------------


def _det(J):
    return torch.linalg.det(J)


def _geometry(X):
    """G (E, dim, n): gradients of the barycentric functions; det (E,)."""
    J = X[:, 1:] - X[:, :1]  # rows: dx of node b
    det = _det(J)
    Ji = torch.linalg.inv(J)  # (E, dim, dim): column b-1 = grad of node b
    G = torch.cat([-Ji.sum(2, keepdim=True), Ji], dim=2)
    return G, det


def _tau(G, uc, nu, dt):
    Gm = G[:, :, 1:]
    g = torch.einsum("erm,erq->emq", Gm, Gm)
    adv = torch.einsum("ea,eab,eb->e", uc, g, uc).abs()
    diff = nu * nu * (g * g).sum((1, 2))
    t = 1.0 / torch.sqrt(4.0 / dt ** 2 + adv + 16.0 * diff)
    bulk = torch.sqrt(4.0 / dt ** 2 + adv + 16.0 * diff) / g.diagonal(dim1=1, dim2=2).sum(1)
    return t, bulk


def _elements(form, dim, dt, X, U, S, NU):
    """Element matrices M (E, n, neq, n, neq) and vectors r (E, n, neq), theta = 1, rho = 1."""
    E, n, neq = X.shape[0], dim + 1, dim + 1
    G, det = _geometry(X)
    V = det / (2.0 if dim == 2 else 6.0)
    nu = NU.mean(1).abs()
    A = X.new_zeros(E, n, neq, n, neq)
    T = X.new_zeros(E, n, neq, n, neq)
    eye = torch.eye(dim, dtype=X.dtype, device=X.device)
    D0 = torch.einsum("eka,ekb->eab", G, G)
    um = U.mean(1)
    if form == "generic":
        tau, bulk = _tau(G, um, nu, dt)
        if dim == 2:
            pts = X.new_tensor([[0.5, 0.5, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5]])
        else:
            a, b = 0.58541019662496845446, 0.13819660112501051518
            pts = X.new_full((4, 4), b) + (a - b) * torch.eye(4, dtype=X.dtype, device=X.device)
        for Nq in pts:
            w = V / len(pts)
            u = torch.einsum("b,ebk->ek", Nq, U)
            adv = torch.einsum("ek,ekb->eb", u, G)
            Sa = Nq[None] + tau[:, None] * adv
            wS = w[:, None] * Sa
            K = w[:, None, None] * nu[:, None, None] * D0 + wS[:, :, None] * adv[:, None, :]
            gam = w[:, None, None] * bulk[:, None, None] * G.transpose(1, 2) + 0.5 * wS[:, :, None] * u[:, None, :]
            A[:, :, :dim, :, :dim] += torch.einsum("eai,ejb->eaibj", gam, G) + torch.einsum("eab,ij->eaibj", K, eye)
            A[:, :, :dim, :, dim] += torch.einsum("ea,eib->eaib", wS, G)
            Sp = w[:, None] * (Nq[None] + 0.5 * tau[:, None] * adv)
            A[:, :, dim, :, :dim] += torch.einsum("ea,ejb->eabj", Sp, G) + \
                torch.einsum("e,eja,eb->eabj", w * tau, G, adv)
            A[:, :, dim, :, dim] += (w * tau)[:, None, None] * D0
            T[:, :, :dim, :, :dim] += torch.einsum("ea,b,ij->eaibj", wS, Nq, eye)
            T[:, :, dim, :, :dim] += torch.einsum("e,eja,b->eabj", w * tau, G, Nq)
    else:
        us = S[:, :, :dim].mean(1)
        tau, bulk = _tau(G, us, nu, dt)
        nrm = G.transpose(1, 2) * (dim * V)[:, None, None]  # (E, n, dim): inward scaled normals
        q = 1.0 / (dim * dim * V)
        un = torch.einsum("ek,eak->ea", um, nrm)
        c1 = 1.0 / (dim * (dim + 1))
        fu = 0.5 * (c1 + (tau * q)[:, None] * un)  # skew half
        uw = um.clone()
        if dim == 3:
            uw[:, 2] = um[:, 1]  # the reference's tetrahedra take v where w is meant here
        dot = torch.einsum("eak,ebk->eab", nrm, nrm)
        diag = c1 * un[:, None, :] + (tau * q)[:, None, None] * un[:, :, None] * un[:, None, :] + \
            (nu * q)[:, None, None] * dot
        Auu = torch.einsum("eab,ij->eaibj", diag, eye)
        Auu = Auu + torch.einsum("ea,ei,ebj->eaibj", fu, uw, nrm)
        nn = torch.einsum("eai,ebj->eaibj", nrm, nrm)
        third = 1.0 / 3.0
        Auu = Auu + (nu * q * third)[:, None, None, None, None] * nn + (bulk * q)[:, None, None, None, None] * nn
        A[:, :, :dim, :, :dim] = Auu
        A[:, :, :dim, :, dim] = torch.einsum("ea,ebi->eaib", c1 + (tau * q)[:, None] * un, nrm)
        A[:, :, dim, :, :dim] = torch.einsum("e,eb,eaj->eabj", tau * q, un, nrm) + \
            0.5 * torch.einsum("e,ea,ebj->eabj", tau * q, torch.einsum("ek,eak->ea", uw, nrm), nrm) + \
            c1 * nrm[:, None, :, :]
        A[:, :, dim, :, dim] = (tau * q)[:, None, None] * dot
        mass = (V / ((dim + 1) * (dim + 2)))[:, None, None] * \
            (1.0 + torch.eye(n, dtype=X.dtype, device=X.device))[None]
        Tuu = mass + (tau / (dim * (dim + 1)))[:, None, None] * un[:, :, None]
        T[:, :, :dim, :, :dim] = torch.einsum("eab,ij->eaibj", Tuu, eye)
        T[:, :, dim, :, :dim] = torch.einsum("e,eaj->eaj", tau * c1, nrm)[:, :, None, :].expand(E, n, n, dim)
    r = -torch.einsum("eaibj,ebj->eai", A, S)
    return A + T / dt, r


def _system(case, pb, up, uadv, chunk=400_000):
    """The conditioned system as node blocks: (start, adj, blocks (nb, neq, neq), rhs (N, neq))."""
    dim, dt = case["dim"], case["dt"]
    neq, dev = dim + 1, up.device
    conn = torch.as_tensor(pb["conn"].astype(np.int64), device=dev)
    X, nu = torch.as_tensor(pb["coords"], device=dev), torch.as_tensor(pb["nu"], device=dev)
    N = len(X)
    pairs = []
    for part in conn.split(chunk):
        pairs.append(torch.unique((part[:, :, None] * N + part[:, None, :]).reshape(-1)))
    keys = torch.unique(torch.cat(pairs))
    blocks = X.new_zeros(len(keys), neq, neq)
    rhs = X.new_zeros(N, neq)
    for part in conn.split(chunk):
        M, r = _elements(case["form"], dim, dt, X[part], uadv[part], up[part], nu[part])
        k = torch.searchsorted(keys, (part[:, :, None] * N + part[:, None, :]).reshape(-1))
        blocks.index_add_(0, k, M.permute(0, 1, 3, 2, 4).reshape(-1, neq, neq))
        rhs.index_add_(0, part.reshape(-1), r.reshape(-1, neq))
    rows, adj = keys // N, keys % N
    # symmetric Dirichlet: the first value of a dof moves its column, the last sets its row
    nodes, comps, vals = (np.asarray(v) for v in pb["bc"])
    dof = nodes.astype(np.int64) * neq + comps
    first, last = np.full(N * neq, np.nan), np.full(N * neq, np.nan)
    first[dof[::-1]] = vals[::-1]
    for c in range(neq):  # numpy keeps the last of repeated assignments
        last[dof[comps == c]] = vals[comps == c]
    first, last = (torch.as_tensor(v, device=dev).reshape(N, neq) for v in (first, last))
    on = ~torch.isnan(first)
    old = up[:, :neq]
    vf = torch.where(on, first - old, torch.zeros_like(old))
    rhs.index_add_(0, rows, -torch.einsum("kij,kj->ki", blocks, vf[adj]))
    rhs = torch.where(on, last - old, rhs)
    blocks = torch.where(on[rows][:, :, None] | on[adj][:, None, :], torch.zeros_like(blocks), blocks)
    at = torch.nonzero(rows == adj)[:, 0]
    blocks[at] += torch.diag_embed(on.to(blocks.dtype))
    start = torch.searchsorted(rows, torch.arange(N + 1, device=dev))
    return start, rows, adj, blocks, rhs


def _csr(start, rows, blocks):
    """Block values in the point-CSR order: row r of a node holds (slot, component)."""
    neq = blocks.shape[1]
    S = (start[1:] - start[:-1])[rows]
    slot = torch.arange(len(rows), device=rows.device) - start[:-1][rows]
    r = torch.arange(neq, device=rows.device)
    pos = neq * neq * start[:-1][rows][:, None, None] + \
        (r[None, :, None] * S[:, None, None] + slot[:, None, None]) * neq + r[None, None, :]
    out = blocks.new_empty(blocks.numel())
    out[pos.reshape(-1)] = blocks.reshape(-1)
    return out


def exact(case, seed):
    dim, neq = case["dim"], case["dim"] + 1
    if case["kind"] == "semi" or (case["kind"] == "step" and max(_counts(case, m)[0] for m in range(case["members"])) * neq > 14000):
        return None  # the whole scheme, or a dense solve of more than 14,000 unknowns
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    out = []
    for m in range(case["members"]):
        pb = _problem(case, seed, m)
        up, lin = torch.as_tensor(pb["up"], device=dev), torch.as_tensor(pb["lin"], device=dev)
        u1, u2, u3 = lin[:, dim:2 * dim], lin[:, 2 * dim:3 * dim], lin[:, 3 * dim:]
        for _ in range(case.get("steps", 1)):
            uadv = 2.1875 * up[:, :dim] - 2.1875 * u1 + 1.3125 * u2 - 0.3125 * u3
            start, rows, adj, blocks, rhs = _system(case, pb, up, uadv)
            if case["kind"] == "assemble":
                out.append({"values": _csr(start, rows, blocks), "rhs": rhs.reshape(-1)})
                break
            N = len(up)
            dense = up.new_zeros(N, neq, N, neq)
            dense[rows, :, adj, :] = blocks
            d = torch.linalg.solve(dense.reshape(N * neq, N * neq), rhs.reshape(-1)).reshape(N, neq)
            u3, u2, u1 = u2, u1, up[:, :dim]
            up = up + d
        else:
            out.append({"solution": up, "linearized": torch.cat([uadv, u1, u2, u3], dim=1)})
    return out
