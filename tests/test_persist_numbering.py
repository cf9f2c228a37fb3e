"""One-launch Krylov solves (csrc/persist.cu) of meshes numbered at random, where a block
touches several times as many nodes as with natural numbering and its coarse corrections
come from all over: clusters, the grid with all its values in shared memory and with few.

Bounds: a solve's residual, recomputed on the host, is within the tolerance and the two
evaluations' rounding (200 eps |A||x|).  Time steps of one mesh under two numberings
differ by the solves' tolerance times the condition number of the pressure matrix, about
n^2 for n cells a side."""
import numpy as np
import pytest

from coolfluid3_b200 import NavierStokes, NavierStokesSemiImplicit
from coolfluid3_b200 import problems as P

pytestmark = pytest.mark.gpu


def scattered(pb, seed=5):
    """The problem with its nodes and elements in random order: node i becomes new[i]."""
    rng = np.random.default_rng(seed)
    new = rng.permutation(len(pb.coords)).astype(np.uint32)
    old = np.argsort(new)
    return new, dict(coords=pb.coords[old], conn=new[pb.conn][rng.permutation(len(pb.conn))], up=pb.up[old],
                     lin=pb.lin[old], nu=np.broadcast_to(pb.nu, len(old))[old], bc_nodes=new[pb.bc_nodes])


@pytest.mark.parametrize("dim,n", [(2, 12), (2, 52), (2, 64), (2, 131), (2, 220), (3, 4), (3, 9), (3, 12), (3, 20),
                                   (3, 27)])
@pytest.mark.parametrize("precond", ["jacobi", "two_level_coupled"])
@pytest.mark.parametrize("mixed", [False, True])
def test_solve_of_a_scattered_mesh(dim, n, precond, mixed):
    pb = P.make_problem(dim, n)
    _, q = scattered(pb)
    ns = NavierStokes(q["coords"], q["conn"], dt=pb.dt, use_specializations=False)
    ns.set_state(q["up"], q["lin"], q["nu"])
    ns.add_dirichlet(q["bc_nodes"], pb.bc_comps, pb.bc_values)
    ns.assemble()
    ns.apply_dirichlet()
    tol = 1e-9
    st = ns.solve(precond=precond, tol=tol, max_iters=6000, mixed=mixed, max_refine=40)
    assert st["converged"] == 1
    rp, ci = ns.csr()
    v, b = ns.system()
    x = ns.solution()
    r = np.linalg.norm(b - np.add.reduceat(v * x[ci], rp[:-1]))
    assert r <= tol * np.linalg.norm(b) + 200 * 2.3e-16 * np.linalg.norm(np.add.reduceat(np.abs(v * x[ci]), rp[:-1]))
    ns.close()


@pytest.mark.parametrize("dim,n", [(2, 60), (2, 150), (3, 8), (3, 20)])
def test_semi_implicit_step_of_a_scattered_mesh(dim, n):
    """Two steps (CG with point Jacobi and with the pressure's coarse space) under natural and
    random numbering."""
    pb = P.make_problem(dim, n)
    new, q = scattered(pb)
    tol, out = 1e-12, []
    for coords, conn, u, bc in ((pb.coords, pb.conn, pb.up, pb.bc_nodes), (q["coords"], q["conn"], q["up"], q["bc_nodes"])):
        si = NavierStokesSemiImplicit(coords, conn, dt=pb.dt, theta=0.5)
        si.set_krylov(velocity={"tol": tol}, pressure={"tol": tol})
        si.initial_conditions(u[:, :dim], 1e-2)
        for c in range(dim):
            on = pb.bc_comps == c
            si.add_velocity_dirichlet(bc[on], c, pb.bc_values[on])
        on = pb.bc_comps == dim
        si.add_pressure_dirichlet(bc[on], pb.bc_values[on])
        si.step(2)
        out.append(si.state[0])
        si.close()
    a, b = out[0], out[1][new]
    assert np.linalg.norm(a - b) <= 10 * n * n * tol * np.linalg.norm(a)
