"""One-launch Krylov solves (csrc/persist.cu) that take several launches, or whose grid
barrier runs out of time."""
import ctypes

import numpy as np
import pytest

from coolfluid3_b200 import NavierStokes, NavierStokesSemiImplicit, UfemError, _native
from coolfluid3_b200 import problems as P

pytestmark = pytest.mark.gpu


def system(dim, n, **kw):
    pb = P.make_problem(dim, n)
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False, **kw)
    ns.set_state(pb.up, pb.lin, pb.nu)
    ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
    ns.assemble()
    ns.apply_dirichlet()
    return ns


def stick_barriers(ns, on):
    f = _native.lib().ufem_ns_stick_barriers
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_int], None
    f(ns._h, on)


@pytest.mark.parametrize("precond", ["jacobi", "two_level_coupled"])
def test_a_barrier_that_runs_out_ends_the_solve_with_an_error(precond):
    """96 x 96 cells (the grid form).  A barrier that waits in vain gives up after some
    seconds, which ends its launch and those queued behind it (the solve before took more
    than one), the call fails, and the next solve gives the bits of the first."""
    ns = system(2, 96)
    start = ns.solution()
    kr = dict(precond=precond, tol=1e-11, max_iters=6000)
    st = ns.solve(**kr)
    x = ns.solution()
    assert precond != "jacobi" or st["iterations"] > 256
    ns.set_solution(start)
    stick_barriers(ns, 1)
    with pytest.raises(UfemError, match="barrier"):
        ns.solve(**kr)
    stick_barriers(ns, 0)
    ns.set_solution(start)
    again = ns.solve(**kr)
    assert again["iterations"] == st["iterations"]
    assert np.array_equal(ns.solution(), x)
    ns.close()


def launch_iterations(f, handle, iters):
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_int], None
    f(handle, iters)


@pytest.mark.parametrize("dim,n", [(2, 20), (2, 96), (3, 8), (3, 16)])
@pytest.mark.parametrize("precond", ["jacobi", "two_level_coupled"])
@pytest.mark.parametrize("mixed", [False, True])
def test_bicgstab_over_several_launches(dim, n, precond, mixed):
    """Clusters (20^2, 8^3) and the grid (96^2, 16^3): up to 24 iterations (fewer where an
    inner solve of the mixed form ends), 7 a launch and all in one.  The vectors and scalars of the state are stored as they are, so the bits are the
    same, except for the grid with a coarse space: its first restriction after a launch
    reads r and q where the others sum the terms they are made of, which differs by
    roundings (eps), amplified by less than 1e6 in so few iterations."""
    ns = system(dim, n)
    start = ns.solution()
    kr = dict(precond=precond, tol=1e-13, max_iters=24, raise_on_failure=False, mixed=mixed, max_refine=1)
    out = []
    for per in (256, 7):
        launch_iterations(_native.lib().ufem_ns_launch_iterations, ns._h, per)
        ns.set_solution(start)
        st = ns.solve(**kr)
        out.append((ns.solution(), st["iterations"]))
    (x, it), (y, jt) = out
    assert it == jt > 7  # more than one launch
    if precond == "jacobi" or n in (20, 8):
        assert np.array_equal(x, y)
    else:
        assert np.linalg.norm(x - y) <= 1e-9 * np.linalg.norm(x)
    ns.close()


@pytest.mark.parametrize("dim,n", [(2, 40), (2, 140), (3, 8), (3, 24)])
def test_cg_over_several_launches(dim, n):
    """A semi-implicit step (CG with point Jacobi and with the pressure's coarse space), 7
    iterations a launch and all in one: clusters to the bit; the grid (140^2, 24^3) within
    the solves' tolerance, 1e-10, times the condition number of the pressure matrix, about
    n^2, since a coarse restriction is made anew after every launch."""
    pb = P.make_problem(dim, n)
    out = []
    for per in (256, 7):
        si = NavierStokesSemiImplicit(pb.coords, pb.conn, dt=pb.dt, theta=0.5)
        launch_iterations(_native.lib().ufem_nssi_launch_iterations, si._h, per)
        si.set_krylov(velocity={"tol": 1e-10}, pressure={"tol": 1e-10})
        si.initial_conditions(pb.up[:, :dim], 1e-2)
        for c in range(dim):
            on = pb.bc_comps == c
            si.add_velocity_dirichlet(pb.bc_nodes[on], c, pb.bc_values[on])
        on = pb.bc_comps == dim
        si.add_pressure_dirichlet(pb.bc_nodes[on], pb.bc_values[on])
        v, p = si.step(1)
        assert p["iterations"] > 14
        out.append((si.state[0], v["iterations"], p["iterations"]))
        si.close()
    (a, v1, p1), (b, v2, p2) = out
    assert v1 == v2 and abs(p1 - p2) <= 2
    if n in (40, 8):
        assert p1 == p2 and np.array_equal(a, b)
    else:
        assert np.linalg.norm(a - b) <= 1e-10 * n * n * np.linalg.norm(a)
