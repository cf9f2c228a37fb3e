"""Triangles with FP32 elements: groups of rows whose values are written as one run of the
CSR (at most five rows and 32 off-diagonal blocks) and groups that are not (more rows, as
along a strip, or one node with many neighbours), alone and in a batch.

Oracle and bounds: the FP64 oracle's assembly, with the FP32 bounds of
test_assembly_lists.py (2e-5 of a CSR row's largest entry, 1e-4 of the RHS)."""
import numpy as np
import pytest

from coolfluid3_b200 import Batch, NavierStokes
from coolfluid3_b200 import problems as P

from .test_assembly_lists import check, fields

pytestmark = pytest.mark.gpu


def strip(nx, ny):
    """nx x ny cells of two triangles on a sheared rectangle."""
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="xy")
    coords = np.stack([i + 0.3 * j, 1.1 * j], -1).reshape(-1, 2) / max(nx, ny)
    c = (np.arange(nx)[None, :] + (nx + 1) * np.arange(ny)[:, None]).ravel()
    a, b, d, e = c, c + 1, c + nx + 1, c + nx + 2
    return coords, np.concatenate([np.stack([a, b, e], 1), np.stack([a, e, d], 1)])


def fan(m):
    """m triangles around one node, every other spoke prolonged by a further triangle."""
    t = np.linspace(0.0, 2.0 * np.pi, m, endpoint=False)
    ring = np.stack([np.cos(t), np.sin(t)], 1)
    k = np.arange(m)
    conn = np.stack([np.zeros(m, int), 1 + k, 1 + (k + 1) % m], 1)
    out = k[::2]
    tip = 1 + m + np.arange(len(out))
    more = np.stack([1 + (out + 1) % m, 1 + out, tip], 1)
    mid = 0.5 * (ring[out] + ring[(out + 1) % m])
    return np.vstack([[[0.0, 0.0]], ring, 1.8 * mid]), np.concatenate([conn, more])


MESHES = [strip(1, 1), strip(40, 1), strip(2, 2), strip(9, 9), strip(33, 7), fan(5), fan(16), fan(31), fan(40)]


@pytest.mark.parametrize("mesh", range(len(MESHES)))
@pytest.mark.parametrize("spec", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_groups_written_as_runs_and_otherwise(mesh, spec, precision):
    for warps in (2, 8):
        check(*MESHES[mesh], spec=spec, precision=precision, variant=("warp", warps))


@pytest.mark.parametrize("spec", [False, True])
def test_batch_members_equal_their_own_handles(spec):
    """FP32 members of every kind in one batch, to 1e-6 of a row's largest entry (the element
    code is compiled twice, so it may round differently; FP32 eps is 6e-8)."""
    def member(mesh):
        coords, conn = mesh
        ns = NavierStokes(coords, conn, dt=0.01, use_specializations=spec, precision="fp32")
        ns.set_state(*fields(coords))
        ns.add_dirichlet(np.array([0]), 2, np.zeros(1))
        return ns

    ms, alone = [member(m) for m in MESHES], [member(m) for m in MESHES]
    b = Batch(ms)
    b.assemble()
    for m, a in zip(ms, alone):
        a.assemble()
        a.apply_dirichlet()
        v, r = m.system()
        w, q = a.system()
        rp, _ = a.csr()
        scale = np.maximum.reduceat(np.abs(w), rp[:-1])
        assert np.all(np.maximum.reduceat(np.abs(v - w), rp[:-1]) <= 1e-6 * scale)
        assert np.linalg.norm(r - q) <= 1e-6 * np.linalg.norm(q)


@pytest.mark.parametrize("n", [2, 21])
def test_fp32_copy_of_the_values(n):
    """The FP32 copy is what the inner solves of a mixed solve read: with another matrix the
    refinement would not reach 1e-11."""
    pb = P.make_problem(2, n)
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False, precision="fp32")
    ns.set_state(pb.up, pb.lin, pb.nu)
    ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
    ns.assemble()
    ns.apply_dirichlet()
    st = ns.solve(precond="jacobi", tol=1e-11, mixed=True, max_refine=8, max_iters=4000)
    assert st["converged"] == 1
    ns.close()
