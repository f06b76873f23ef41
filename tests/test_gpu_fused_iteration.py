"""The fused iteration (ofg_step, one CUDA graph) against the same iteration
task by task: the graph runs some levels and reductions inside other kernels or
beside them, the tasks one after the other -- the same arithmetic per cell in the
same order, so the same bits."""
import numpy as np
import pytest

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import LUSGS_SEQUENCE, NS_SOLVER, TURB_SOLVER, Batch, Solver
from oneflow_b200.walldist import plate_wall_distance

pytestmark = pytest.mark.gpu


def case(name):
    if name == "plate3d":
        m = meshgen.flat_plate_tets(16, 10, 6)
        m.wall_dist = plate_wall_distance(m)
        return m, P.rans_plate(sweep_order=1)
    if name == "plate3d_fp64":
        m = meshgen.flat_plate_tets(9, 7, 5)
        m.wall_dist = plate_wall_distance(m)
        return m, P.rans_plate(sweep_order=1, precision=0, igrad=0, venkat_kh3=0, vencat_coef=0.0001)
    if name == "plate2d_natural":
        return meshgen.plate_2d(40, 30), P.defaults(vismodel=1, ischeme=12, reynolds=1e4, cflst=1.0, cfled=5.0)
    ni, nj, prec, ilim = {"bump_tiny": (3, 2, 0, -1), "bump_limited": (61, 37, 1, 2), "bump_fp64": (64, 32, 0, 2)}[name]
    return (meshgen.bump_channel(ni, nj),
            P.euler_bump(precision=prec, sweep_order=1, ilim=ilim, vencat_coef=0.05, cflst=1.0, cfled=5.0, ncfl=3))


@pytest.mark.parametrize("name", ["bump_tiny", "bump_limited", "bump_fp64", "plate2d_natural", "plate3d", "plate3d_fp64"])
def test_fused_iterations_are_the_tasks(name):
    m, prm = case(name)
    a, b = Solver(m, prm), Solver(m, prm)
    a.init_flowfield()
    b.init_flowfield()
    tids = [NS_SOLVER] + ([TURB_SOLVER] if prm.vismodel >= 3 else [])
    norms = []
    for it in range(5):
        if it in (0, 1, 3):   # steps of one, two and two iterations: the state between calls is carried too
            a.step(1 if it == 0 else 2)
        b.set_outer_step(it + 1)
        for tid in tids:
            for t in LUSGS_SEQUENCE:
                b.task(t, tid)
            if tid == NS_SOLVER:
                norms.append(b.residual_norms())
    assert np.array_equal(a.state(), b.state())
    assert np.array_equal(a.res_history(), np.array(norms))
    if prm.vismodel >= 3:
        assert np.array_equal(a.state(TURB_SOLVER), b.state(TURB_SOLVER))


@pytest.mark.parametrize("name", ["plate3d", "plate3d_fp64"])
def test_overlapped_iterations_are_the_whole_ones(name):
    """ofg_step runs the next gradients beside the SA stage; a batch runs whole
    iterations.  State, forces and the gradient records agree bit for bit after
    calls of one, two and three iterations, and when the two alternate."""
    m, prm = case(name)
    a, b = Solver(m, prm), Solver(m, prm)
    a.init_flowfield()
    b.init_flowfield()
    batch, own = Batch([b]), Batch([a])
    for n, whole in ((1, False), (2, False), (3, False), (1, True), (2, False)):
        (own if whole else a).step(n)
        batch.step(n)
        assert np.array_equal(a.state(), b.state())
        assert np.array_equal(a.state(TURB_SOLVER), b.state(TURB_SOLVER))
        assert np.array_equal(a.forces(), b.forces())
        for field in ("dqdx", "dqdz", "limiter"):
            assert np.array_equal(a.field(field), b.field(field))
    assert np.array_equal(a.res_history(), b.res_history())
    batch.close()
    own.close()
