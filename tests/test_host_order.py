"""What the library's host code asks of the device and in which order, on the CPU: each
test runs in a child process whose CUDA runtime is tests/fake_cudart.cpp."""
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="session")
def runtime(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-I",
                    os.path.join(ROOT, "coolfluid3_b200", "csrc"), os.path.join(HERE, "fake_cudart.cpp"), "-o", so],
                   check=True)
    return so


PREAMBLE = """
import ctypes, sys
import numpy as np
from coolfluid3_b200 import Batch, NavierStokes, NavierStokesSemiImplicit, UfemError
from coolfluid3_b200 import problems as P
fake = ctypes.CDLL(sys.argv[1])
STREAM = 4096  # any stream but the legacy one

def solver(dim, n, **kw):
    pb = P.make_problem(dim, n)
    ns = NavierStokes(pb.coords, pb.conn, dt=pb.dt, use_specializations=False, **kw)
    ns.set_state(pb.up, pb.lin, pb.nu)
    ns.add_dirichlet(pb.bc_nodes, pb.bc_comps, pb.bc_values)
    return ns, pb

def check(what):
    assert fake.fake_faults() == 0, what + ": a stream was given work beside an upload in flight"
    assert fake.fake_pending() == 0, what + ": returned with an upload in flight"
"""


def run(runtime, body):
    env = dict(os.environ, LD_PRELOAD=runtime, PYTHONPATH=ROOT)
    p = subprocess.run([sys.executable, "-c", PREAMBLE + textwrap.dedent(body), runtime], env=env, cwd=ROOT,
                       capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stdout + p.stderr


def test_uploads_land_before_other_streams_read_them(runtime, tmp_path):
    """The static lists, condition plans, batch tables, coarse spaces and solutions that
    calls upload: nothing of them is in flight when another stream is given work or
    the call returns."""
    run(runtime, f"""
    ns, pb = solver(2, 12)
    check("create")
    ns.add_dirichlet_function(pb.bc_nodes[:3], 0, "x*t")
    ns.add_neumann(pb.conn[:1, :2].astype(np.uint32), 2, 0.5)
    ns.assemble(STREAM)
    ns.apply_dirichlet(STREAM)
    check("conditions")
    for kr in (dict(precond="jacobi"), dict(precond="two_level_coupled"), dict(method="gmres", precond="jacobi")):
        ns.prepare_solve(**kr)
        check("prepare_solve")
        ns.solve(STREAM, raise_on_failure=False, max_iters=4, **kr)
        check("solve")
    ns.set_solution(np.ones(ns.nb_rows))
    check("set_solution")
    ns.write_restart(r"{tmp_path}/r.cfg", time_step=0.1)
    ns.read_restart(r"{tmp_path}/r.cfg")
    check("read_restart")

    members = [solver(2, n)[0] for n in (6, 9)]
    b = Batch(members)
    check("batch")
    for pre in ("jacobi", "two_level_coupled"):
        b.assemble(STREAM)
        check("batch assemble")
        b.solve(STREAM, precond=pre, max_iters=4)
        check("batch solve")
    b.set_active([True, False])
    b.assemble(STREAM)
    check("batch with a held member")

    for dim, n in ((2, 20), (3, 8)):
        pb = P.make_problem(dim, n)
        si = NavierStokesSemiImplicit(pb.coords, pb.conn, dt=pb.dt, theta=0.5)
        check("semi-implicit create")
        si.initial_conditions(pb.up[:, :dim], 1e-2)
        si.add_velocity_dirichlet(pb.bc_nodes[:4], 0, np.zeros(4))
        si.add_pressure_dirichlet(np.array([0]), np.zeros(1))
        check("semi-implicit conditions")
        si.step(2, stream=STREAM)
        check("semi-implicit step")
    """)


def test_a_late_barrier_of_any_launch_is_an_error(runtime):
    """A solve expected to take 600 iterations queues three launches (80 x 80 cells: the
    grid form) before the host looks: a barrier that ran out of time in the first, a
    middle or the last of them is an error, and the solve after it starts afresh."""
    run(runtime, """
    ns, pb = solver(2, 80)
    ns.assemble(STREAM)
    ns.apply_dirichlet(STREAM)
    kr = dict(precond="jacobi", max_iters=3000)
    for late in (0, 1, 2):
        fake.fake_solves(600, -1)
        assert ns.solve(STREAM, **kr)["iterations"] == 600
        fake.fake_solves(600, late)
        try:
            ns.solve(STREAM, **kr)
        except UfemError as e:
            assert "barrier" in str(e)
        else:
            raise AssertionError(f"launch {late} was late and the solve succeeded")
        assert fake.fake_launches() == 3
    """)


@pytest.mark.parametrize("precond", ["jacobi", "two_level_coupled"])
def test_a_system_is_planned_once(runtime, precond):
    """The plan of a one-launch solve (a walk over the graph on the host) is made by
    prepare_solve, and by nothing after it: not the first solve, not a solve without
    allocation, not a new batch with the same members."""
    run(runtime, f"""
    from coolfluid3_b200 import _native, krylov_options
    kr = dict(precond="{precond}", max_iters=20)
    ns, _ = solver(2, 80)
    ns.prepare_solve(**kr)
    assert fake.fake_plans() == 1
    ns.assemble()
    ns.apply_dirichlet()
    ns.solve(**kr)
    assert fake.fake_plans() == 0
    st = _native.KrylovStatus()
    plain = krylov_options(precond="jacobi", max_iters=20)
    for k in range(3):
        _native.lib().ufem_ns_solve_noalloc(ns.handle, ctypes.byref(plain), ctypes.byref(st), None)
    assert fake.fake_plans() == (0 if "{precond}" == "jacobi" else 1)

    for mixed in (False, "matrix_free"):
        ms = [solver(2, n)[0] for n in (8, 80)]
        for m in ms:
            m.prepare_solve(batched=True, mixed=mixed, **kr)
        assert fake.fake_plans() == 2
        for k in range(2):
            b = Batch(ms)
            b.assemble()
            b.solve(mixed=mixed, **kr)
            b.close()
        assert fake.fake_plans() == 0
    """)


def test_batch_members_of_both_forms_run_beside_each_other(runtime):
    """Members that fit a cluster and members that do not, in one batch: the clusters go to
    streams of their own and the others' iterations are given to the caller's stream
    before the host waits for anything; without such others the largest clusters run on
    the caller's stream."""
    run(runtime, """
    fake.fake_log.restype = ctypes.c_char_p
    kr = dict(precond="jacobi", max_iters=8)
    def log(sizes):
        b = Batch([solver(2, n)[0] for n in sizes])
        b.assemble(STREAM)
        fake.fake_log()
        b.solve(STREAM, **kr)
        return fake.fake_log().decode()
    both = log([6, 140, 20])
    first = min(both.index(c) for c in "cC" if c in both)
    assert "C" not in both
    assert "G" in both[first:].split("S")[0], both
    small = log([6, 20])
    assert "C" in small and "G" not in small.split("C")[1].split("S")[0], small
    """)


def test_creation_does_not_free(runtime):
    """Building a handle does not hold up what other threads have on the device: it frees
    nothing (a free waits for all of it)."""
    run(runtime, """
    fake.fake_frees()
    kept = [solver(dim, n, precision=p) for dim, n in ((2, 12), (3, 5)) for p in ("fp64", "fp32")]
    assert fake.fake_frees() == 0
    """)


def test_a_device_without_room_for_a_cluster_solves_on_the_grid(runtime):
    """A system that would take one cluster goes to the grid where the device cannot run the
    cluster, and a batch's members to the chunk kernels."""
    run(runtime, """
    fake.fake_log.restype = ctypes.c_char_p
    def solved(clusters):
        fake.fake_clusters(clusters)
        ns, _ = solver(2, 12)
        ns.assemble(STREAM)
        ns.apply_dirichlet(STREAM)
        fake.fake_log()
        ns.solve(STREAM, precond="jacobi")
        one = fake.fake_log().decode()
        b = Batch([solver(2, 12)[0]])
        b.assemble(STREAM)
        b.solve(STREAM, precond="jacobi", max_iters=8)
        return one, fake.fake_log().decode()
    one, batch = solved(8)
    assert "P" in one and "C" in batch and "G" not in batch
    one, batch = solved(0)
    assert "R" in one and "P" not in one and "C" not in batch and "G" in batch
    """)
