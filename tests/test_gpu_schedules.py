"""The sweep schedule among a context's other choices: the autotuner times the
level kernels' shapes with level launches whatever the context came with; a
schedule that is not in use holds no memory; a second mesh uploaded into a
context tuned to the chained sweeps; chained contexts made and dropped by several
threads at once.  The overlapped SA iteration of calls of ten and more: against
whole iterations, and around a caller's stream."""
import threading

import numpy as np
import pytest
import torch

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import TURB_SOLVER, Batch, Solver
from oneflow_b200.walldist import plate_wall_distance

pytestmark = pytest.mark.gpu


def plate(nx, ny, nz, order, precision=1):
    m = meshgen.flat_plate_tets(nx, ny, nz)
    m.wall_dist = plate_wall_distance(m)
    return m, P.rans_plate(precision=precision, sweep_order=order)


@pytest.mark.parametrize("came", [1, 0])
def test_the_autotuner_times_level_shapes_with_level_launches(came):
    m, prm = plate(23 + came, 11, 7, 0)   # a mesh of its own: no cached choice
    s = Solver(m, prm)
    assert s.tuning()["sweep_persistent"] == 1   # natural order
    if not came:
        s.set_tuning(sweep_persistent=0)
    s.init_flowfield()
    before, reps = s.counters()[1], 3
    t = s.autotune(reps=reps)
    lower, upper = s.sweep_levels()
    shapes, sweep, chained = 6, lower + upper - 1, 4   # the upper sweep's first level is not launched
    gathers = (8 + 6) * reps
    extra = s.counters()[1] - before - (shapes * sweep + chained) * reps - gathers
    assert 0 <= extra < 30   # the launches that fill the timed groups' inputs once
    assert 0.0 < t["ms_tuned"] <= t["ms_default"]
    assert t["sweep_persistent"] in (0, 1)
    s.step(2)
    assert np.isfinite(s.state()).all()


def test_a_schedule_that_is_not_in_use_holds_no_memory():
    s = Solver(meshgen.bump_channel(200, 100), P.euler_bump(sweep_order=0))   # about 300 levels of 130 cells: chained
    assert s.tuning()["sweep_persistent"] == 1
    free = []
    for chained in (1, 0, 1, 0):
        s.set_tuning(sweep_persistent=chained)
        free.append(torch.cuda.mem_get_info()[0])
    # 60,000 edges a sweep, in both at 20 bytes, in the scratch at 120
    assert free[0] < free[1] - (8 << 20) and free[2:] == free[:2]


@pytest.mark.parametrize("order", [0, 1])
def test_a_second_mesh_in_a_context_tuned_to_chained(order):
    def fresh(m, prm):
        s = Solver(m, prm)
        s.set_tuning(sweep_persistent=1)
        return s

    def go(s):
        s.init_flowfield()
        s.step(3)
        return [s.state(), s.state(TURB_SOLVER)]

    (a, prm), (b, _) = plate(14, 9, 5, order), plate(20, 8, 6, order)
    want = go(fresh(b, prm))
    s = fresh(a, prm)
    first = go(s)
    for m, ref in ((b, want), (a, first)):
        s._keep, s.mesh, s.nT = m.as_arrays(), m, m.n_cells + m.n_bfaces
        k = s._keep
        s._check(s.L.ofg_upload_mesh(s.h, m.n_nodes, k["x"], k["y"], k["z"], m.n_faces, k["fnc"], k["fn"], k["lc"],
                                     k["rc"], m.n_cells, m.n_bfaces, k["bct"], k["wd"].ctypes.data))
        assert s.tuning()["sweep_persistent"] == 1
        assert all(np.array_equal(x, y) for x, y in zip(go(s), ref))


@pytest.mark.parametrize("order,precision", [(0, 1), (1, 1), (1, 0)])
def test_a_callers_stream_around_the_overlapped_iteration(order, precision):
    m, prm = plate(16, 10, 6, order, precision)
    a, b = Solver(m, prm), Solver(m, prm)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    big = torch.empty(1 << 26, device="cuda")
    a.init_flowfield()
    b.init_flowfield()
    for k, n in enumerate((1, 10, 12, 11)):   # the caller's streams in turn, then the context's own again
        if k < 3:
            st = streams[k % 2]
            b.set_stream(st.cuda_stream)
            with torch.cuda.stream(st):
                big.add_(1.0)   # the caller's own work ahead of the call
        else:
            b.set_stream(0)
        a.step(n)
        b.step(n)
        assert np.array_equal(a.state(), b.state())
        assert np.array_equal(a.state(TURB_SOLVER), b.state(TURB_SOLVER))
        assert np.array_equal(a.field("dqdx"), b.field("dqdx"))
    assert np.array_equal(a.res_history(), b.res_history())


@pytest.mark.parametrize("order,precision,igrad", [(1, 1, 2), (1, 1, 0), (0, 1, 0), (1, 0, 0), (0, 0, 2)])
def test_overlapped_calls_are_the_whole_iterations(order, precision, igrad):
    """Calls long enough to be overlapped, shorter ones and odd and even numbers of
    iterations between them, against a batch of the one solve, which runs whole ones."""
    m, prm = plate(12, 9, 5, order, precision)
    prm.igrad = igrad
    a, b = Solver(m, prm), Solver(m, prm)
    a.init_flowfield()
    b.init_flowfield()
    batch = Batch([b])
    for n in (10, 1, 11, 2, 12):
        a.step(n)
        batch.step(n)
        assert np.array_equal(a.state(), b.state())
        assert np.array_equal(a.state(TURB_SOLVER), b.state(TURB_SOLVER))
        assert np.array_equal(a.forces(), b.forces())
        for field in ("dqdx", "dqdz", "limiter"):
            assert np.array_equal(a.field(field), b.field(field))
    assert np.array_equal(a.res_history(), b.res_history())
    batch.close()


def test_chained_contexts_of_several_threads():
    m, prm = meshgen.bump_channel(40, 20), P.euler_bump()

    def solve():
        s = Solver(m, prm)
        s.init_flowfield()
        s.step(3)
        return s.state()

    want, bad = solve(), []

    def work():
        try:
            for _ in range(8):
                if not np.array_equal(solve(), want):
                    bad.append("different bits")
        except Exception as e:
            bad.append(e)

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
