"""The Dirichlet pass is one launch over the rows that hold constrained columns and
the constrained rows: block edges of both parts, and either part alone."""
import numpy as np
import pytest

from coolfluid3_b200 import Batch, NavierStokes

from .util import small_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 9), (3, 3)])
@pytest.mark.parametrize("which", ["one", "32", "33", "all"])
@pytest.mark.parametrize("batched", [False, True])
def test_constrained_sets_of_any_size(dim, n, which, batched):
    """The rows and right-hand side of the pass are the sequential form's, term by
    term: from one assembled system (bitwise the same in both handles), the
    conditioned one is rebuilt here from the unconditioned one."""
    pb = small_problem(dim, n)
    neq, N = dim + 1, len(pb.coords)
    rng = np.random.default_rng(4)
    dofs = rng.permutation(N * neq)[: {"one": 1, "32": 32, "33": 33, "all": N * neq}[which]]
    values = rng.standard_normal(len(dofs))

    def handle(bcs):
        ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False)
        ns.set_state(pb.up, pb.lin, pb.nu)
        if bcs:
            ns.add_dirichlet((dofs // neq).astype(np.int64), (dofs % neq).astype(np.int32), values)
        return ns

    free, ns = handle(False), handle(True)
    free.assemble()
    if batched:
        b = Batch([ns])
        b.assemble()
    else:
        ns.assemble()
        ns.apply_dirichlet()
    rp, ci = free.csr()
    v, rhs = free.system()
    v, rhs = v.copy(), rhs.copy()
    old = np.asarray(pb.up).reshape(N, -1)[:, :neq].reshape(-1)
    new = np.zeros(N * neq)
    new[dofs] = values - old[dofs]
    fixed = np.zeros(N * neq, dtype=bool)
    fixed[dofs] = True
    order = {d: k for k, d in enumerate(dofs)}
    for r in range(N * neq):
        q = np.arange(rp[r], rp[r + 1])
        if fixed[r]:
            v[q] = (ci[q] == r).astype(float)
            rhs[r] = new[r]
        else:
            for p in sorted(q[fixed[ci[q]]], key=lambda p: order[ci[p]]):
                rhs[r] += -v[p] * new[ci[p]]
                v[p] = 0.0
    gv, grhs = ns.system()
    assert np.array_equal(gv, v)
    assert np.array_equal(grhs, rhs)
    assert np.array_equal(ns.solution()[dofs], new[dofs])
    if batched:
        b.close()
