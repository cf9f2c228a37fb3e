"""Assembly kernels on meshes with linked (periodic) nodes: the static lists of a master
row hold the elements of both sides, and the linked rows between them, which have no
elements, take no part in the groups.  The oracle and the bound are those of
test_assembly_lists.py: 1e-11 of each CSR row's largest entry."""
import numpy as np
import pytest

import oracle as O
from coolfluid3_b200 import NavierStokes
from coolfluid3_b200 import problems as P

from .util import row_scaled_error, vec_rel_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n", [(2, 3), (2, 9), (3, 3), (3, 5)])
@pytest.mark.parametrize("axis", [0, -1])
@pytest.mark.parametrize("spec", [False, True])
def test_linked_faces(dim, n, axis, spec):
    """The faces at the two ends of the first or the last axis linked: linked rows at every
    row's end, or all together at the end."""
    pb = P.make_problem(dim, n)
    step = (n + 1) ** (0 if axis == 0 else dim - 1)
    ids = np.arange((n + 1) ** dim)
    slaves = ids[(ids // step) % (n + 1) == n]
    links = (slaves.astype(np.uint32), (slaves - n * step).astype(np.uint32))
    rng = np.random.default_rng(dim * 100 + n)
    up = rng.normal(size=pb.up.shape)
    lin = np.tile(up[:, :dim], (1, 4)) + 0.1 * rng.normal(size=pb.lin.shape)
    up[links[0]], lin[links[0]] = up[links[1]], lin[links[1]]
    o = O.Oracle(pb.coords, pb.conn, O.options(dt=pb.dt, use_specializations=spec), periodic_links=links)
    o.set_state(up, lin, pb.nu)
    o.assemble()
    ov, orr = o.system()
    rp, _ = o.csr()
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=spec, periodic_links=links)
    ns.set_state(up, lin, pb.nu)
    for variant in [("warp", 2), ("warp", 8), ("chunk", 4)] + ([("warp24", 4)] if dim == 3 else []):
        ns.set_assembly_kernel(*variant)
        ns.assemble()
        v, r = ns.system()
        assert row_scaled_error(v, ov, rp) <= 1e-11, variant
        assert vec_rel_error(r, orr) <= 1e-11, variant
    ns.close()
