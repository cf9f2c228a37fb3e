"""One-launch Krylov solves (csrc/persist.cu) that take several launches, or whose grid
barrier runs out of time."""
import ctypes

import numpy as np
import pytest

from coolfluid3_b200 import NavierStokes, UfemError, _native
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
