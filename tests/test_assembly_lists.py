"""The warp assembly kernel's static lists and reductions where they can go wrong:
slots with one contributor (boundary edges), with more than the seven of an item
word (a spindle of tetrahedra around one edge), rows with more than 16 off-diagonal
blocks, groups of one and of many rows, periodic rows, every tau.

Oracle: the FP64 oracle's assembly; bound 1e-11 of each CSR row's largest entry, the
bound of the element parity tests."""
import numpy as np
import pytest

import oracle as O
from coolfluid3_b200 import Batch, NavierStokes

from .util import row_scaled_error, small_problem, vec_rel_error

pytestmark = pytest.mark.gpu


def fields(coords, seed=3):
    rng = np.random.default_rng(seed)
    n, dim = coords.shape
    up = rng.normal(size=(n, dim + 1))
    lin = np.tile(up[:, :dim], (1, 4)) + 0.1 * rng.normal(size=(n, 4 * dim))
    return np.ascontiguousarray(up), np.ascontiguousarray(lin), np.abs(rng.normal(size=n)) * 0.01 + 1e-3


def spindle(m):
    """m tetrahedra around the edge (0, 1)."""
    a = np.linspace(0.0, 2.0 * np.pi, m, endpoint=False)
    coords = np.vstack([[0.0, 0.0, -1.0], [0.0, 0.0, 1.0], np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(3 * a)], 1)])
    k = np.arange(m)
    return coords, np.stack([np.zeros(m, int), np.ones(m, int), 2 + (k + 1) % m, 2 + k], 1)


def check(coords, conn, *, spec, supg="metric", variant=("warp", 4), precision="fp64"):
    up, lin, nu = fields(coords)
    ns = NavierStokes(coords, conn, dt=0.01, use_specializations=spec, supg_type=supg, precision=precision)
    ns.set_state(up, lin, nu)
    ns.set_assembly_kernel(*variant)
    ns.assemble()
    v, r = ns.system()
    o = O.Oracle(coords, conn, O.options(dt=0.01, use_specializations=spec, supg_type=supg))
    o.set_state(up, lin, nu)
    o.assemble()
    ov, orr = o.system()
    rp, _ = o.csr()
    # FP32 elements: the bounds of the precision's own parity tests
    tv, tr = (1e-11, 1e-11) if precision == "fp64" else (2e-5, 1e-4)
    assert row_scaled_error(v, ov, rp) <= tv
    assert vec_rel_error(r, orr) <= tr
    ns.close()


@pytest.mark.parametrize("m", [3, 7, 8, 15, 24, 25, 32, 33])
@pytest.mark.parametrize("spec", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_edges_with_many_tetrahedra(m, spec, precision):
    coords, conn = spindle(m)
    for variant in (("warp", 2), ("warp24", 4)):
        check(coords, conn, spec=spec, variant=variant, precision=precision)


@pytest.mark.parametrize("dim,n", [(2, 1), (2, 2), (2, 9), (3, 1), (3, 2), (3, 4)])
@pytest.mark.parametrize("supg", ["metric", "tezduyar", "cf2"])
def test_small_meshes_every_tau(dim, n, supg):
    pb = small_problem(dim, n)
    rng = np.random.default_rng(n)
    perm = rng.permutation(pb.nb_nodes)
    coords = pb.coords[np.argsort(perm)]
    conn = perm[pb.conn.astype(np.int64)][rng.permutation(pb.nb_elems)]
    check(coords, conn, spec=False, supg=supg)


def test_batch_of_both_element_routines():
    """Members with METRIC and with another tau in one batch: each the bits it has in
    a batch of its own."""
    def member(supg):
        pb = small_problem(2, 6)
        ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False, supg_type=supg)
        ns.set_state(*fields(pb.coords))
        ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
        return ns

    kinds = ["metric", "tezduyar", "metric", "cf2"]
    ms = [member(k) for k in kinds]
    b = Batch(ms)
    b.assemble()
    for k, m in zip(kinds, ms):
        one = member(k)
        alone = Batch([one])
        alone.assemble()
        for x, y in zip(m.system(), one.system()):
            assert np.array_equal(x, y), k
        alone.close()
    b.close()
