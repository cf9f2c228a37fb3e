"""One-launch Krylov solves (csrc/persist.cu) at the sizes where their layout
changes: one block, clusters of every size, the cooperative grid, values that do
not fit shared memory, rows longer than a warp's pairs, more iterations than one
launch runs.  Each solve's true residual is recomputed on the host from the
system the library returns.

Bound: the library accepts a solve when its own ||b - A x|| <= tol ||b||; the two
evaluations of A x differ by at most about n eps |A||x| per row, n <= 200 terms."""
import numpy as np
import pytest

from coolfluid3_b200 import NavierStokes
from coolfluid3_b200 import problems as P

pytestmark = pytest.mark.gpu


def residual_and_bound(ns, tol):
    rp, ci = ns.csr()
    v, b = ns.system()
    x = ns.solution()
    ax = np.add.reduceat(v * x[ci], rp[:-1])
    mag = np.add.reduceat(np.abs(v * x[ci]), rp[:-1])
    return np.linalg.norm(b - ax), tol * np.linalg.norm(b) + 200 * 2.3e-16 * np.linalg.norm(mag)


def solver(pb, **kw):
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False, **kw)
    ns.set_state(pb.up, pb.lin, pb.nu)
    ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
    ns.assemble()
    ns.apply_dirichlet()
    return ns


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 7), (2, 15), (2, 30), (2, 43), (2, 64), (2, 75), (2, 131),
                                   (3, 1), (3, 3), (3, 6), (3, 9), (3, 13), (3, 20), (3, 31)])
@pytest.mark.parametrize("precond", ["none", "jacobi", "two_level_coupled"])
def test_solve_meets_its_residual(dim, n, precond):
    if precond == "none" and n > 16:
        pytest.skip("unpreconditioned solves of fine meshes do not converge")
    ns = solver(P.make_problem(dim, n))
    tol = 1e-9
    st = ns.solve(precond=precond, tol=tol, max_iters=5000)
    assert st["converged"] == 1 and st["rel_residual"] <= tol
    r, bound = residual_and_bound(ns, tol)
    assert r <= bound, (r, bound)
    it = st["iterations"]
    x = ns.solution()
    ns.set_solution(np.zeros_like(x))  # the Dirichlet pass left the row values in the first guess
    ns.apply_dirichlet()
    st2 = ns.solve(precond=precond, tol=tol, max_iters=5000)
    assert st2["converged"] == 1
    ns.close()
    assert it > 0


@pytest.mark.parametrize("dim,n", [(2, 20), (2, 64), (3, 8), (3, 16)])
def test_mixed_and_repeatable(dim, n):
    """FP32 operator inside FP64 refinement; the same bits from two handles."""
    pb = P.make_problem(dim, n)
    out = []
    for _ in range(2):
        ns = solver(pb)
        st = ns.solve(precond="jacobi", tol=1e-10, max_iters=5000, mixed=True, max_refine=40)
        assert st["converged"] == 1
        r, bound = residual_and_bound(ns, 1e-10)
        assert r <= bound
        out.append(ns.solution())
        ns.close()
    assert np.array_equal(out[0], out[1])


def test_iteration_limit_and_resume():
    """A limit below the need stops at it with status 1; more than one launch's
    iterations (256) continue from the stored state."""
    ns = solver(P.make_problem(2, 96))
    st = ns.solve(precond="jacobi", tol=1e-12, max_iters=10, raise_on_failure=False)
    assert st["converged"] == 0 and st["iterations"] >= 10
    st = ns.solve(precond="jacobi", tol=1e-11, max_iters=6000)
    assert st["converged"] == 1 and st["iterations"] > 256
    r, bound = residual_and_bound(ns, 1e-11)
    assert r <= bound
    ns.close()


@pytest.mark.parametrize("spokes", [20, 50])
def test_long_rows(spokes):
    """A fan: one node with `spokes` neighbours (more than a slice's usual width)."""
    a = np.linspace(0.0, 2.0 * np.pi, spokes, endpoint=False)
    coords = np.vstack([[0.0, 0.0], np.stack([np.cos(a), np.sin(a)], 1)])
    k = np.arange(spokes)
    conn = np.stack([np.zeros(spokes, int), 1 + k, 1 + (k + 1) % spokes], 1)
    ns = NavierStokes(coords, conn, dt=0.05, use_specializations=False)
    u = np.stack([coords[:, 1], -coords[:, 0]], 1)
    ns.initial_conditions(u, 1e-2)
    ns.add_dirichlet(1 + k, 0, 0.3)
    ns.add_dirichlet(1 + k, 1, 0.0)
    ns.add_dirichlet(np.array([1]), 2, 0.0)
    ns.assemble()
    ns.apply_dirichlet()
    st = ns.solve(precond="jacobi", tol=1e-10)
    assert st["converged"] == 1
    r, bound = residual_and_bound(ns, 1e-10)
    assert r <= bound
    ns.close()


def test_zero_right_hand_side():
    """b = 0 returns the zero solution whatever the first guess."""
    pb = P.make_problem(2, 12)
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt)
    z = np.zeros_like(pb.up)
    ns.set_state(z, np.zeros_like(pb.lin), pb.nu)
    ns.add_dirichlet(np.array([0]), 2, 0.0)
    ns.assemble()
    ns.apply_dirichlet()
    ns.set_solution(np.full(ns.nb_rows, 0.5))
    st = ns.solve(precond="jacobi", tol=1e-10)
    assert st["converged"] == 1 and np.all(ns.solution() == 0.0)
    ns.close()


@pytest.mark.parametrize("mixed,precond", [(False, "jacobi"), ("matrix_free", "two_level_coupled")])
def test_batch_members_of_both_forms(mixed, precond):
    """Members solved in one cluster (of several sizes) and a member too large for one
    (131 x 131 cells) in one batch: each the bits it has in a batch of its own, its
    true residual within the tolerance."""
    from coolfluid3_b200 import Batch

    def member(n):
        pb = P.make_problem(2, n)
        ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False,
                          precision="fp32" if mixed else "fp64")
        ns.set_state(pb.up, pb.lin, pb.nu)
        ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
        return ns

    sizes = [4, 131, 12, 40, 25]
    kr = dict(precond=precond, tol=1e-9, max_iters=6000, mixed=mixed)
    ms = [member(n) for n in sizes]
    b = Batch(ms)
    b.assemble()
    st = b.solve(**kr)
    for n, m, s in zip(sizes, ms, st):
        assert s["converged"] == 1 and s["rel_residual"] <= 1e-9, (n, s)
        one = member(n)
        alone = Batch([one])
        alone.assemble()
        s1 = alone.solve(**kr)[0]
        assert s1["iterations"] == s["iterations"]
        assert np.array_equal(one.solution(), m.solution()), n
        alone.close()
        if not mixed:
            r, bound = residual_and_bound(m, 1e-9)
            assert r <= bound
    b.close()
