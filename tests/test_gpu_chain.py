"""The chained LU-SGS sweeps (one launch per sweep, a cluster of blocks running
every level) against one launch per level: the same per-cell arithmetic in the
same dependency order, so the same bits, at the sizes where the schedule can go
wrong: levels of a single cell, fewer levels than the block's groups, levels
wider than one pass of the block or the cluster, neighbours beyond the ring."""
import numpy as np
import pytest

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import Batch, Solver, TURB_SOLVER
from oneflow_b200.walldist import plate_wall_distance

pytestmark = pytest.mark.gpu


def case(name):
    if name.startswith("bump"):   # one block; a cluster of 4; several passes of a block on a colour-major order
        ni, nj, prec, order = {"bump_row": (40, 1, 0, 0), "bump_small": (17, 9, 1, 0), "bump_cluster": (230, 90, 0, 0),
                               "bump_colour": (33, 21, 0, 1)}[name]
        return meshgen.bump_channel(ni, nj), P.euler_bump(precision=prec, sweep_order=order, ilim=2, vencat_coef=0.05)
    if name == "plate2d":
        return meshgen.plate_2d(40, 30), P.defaults(vismodel=1, ischeme=12, reynolds=1e4, cflst=1.0, cfled=5.0)
    if name == "mixed3d":   # up to seven faces a cell
        m = meshgen.bump_box_mixed(8, 6, 6)
        return m, P.defaults(dimension=3, vismodel=1, ischeme=12, ilim=1, reynolds=1e4, visSRModel=1)
    nx, ny, nz, prec = {"plate3d_far": (48, 40, 12, 0), "plate3d_far_mixed": (48, 40, 12, 1)}[name]
    m = meshgen.flat_plate_tets(nx, ny, nz)
    m.wall_dist = plate_wall_distance(m)
    return m, P.rans_plate(precision=prec, sweep_order=0)


def run(s, steps):
    s.step(steps)
    out = [s.state(), s.res_history()]
    return out + [s.state(TURB_SOLVER)] if s.params.vismodel >= 3 else out


@pytest.mark.parametrize("name", ["bump_row", "bump_small", "bump_cluster", "bump_colour", "plate2d", "mixed3d",
                                  "plate3d_far", "plate3d_far_mixed"])
def test_chained_sweeps_give_the_same_bits(name):
    m, prm = case(name)
    got = []
    for chained in (0, 1):
        s = Solver(m, prm)
        s.set_tuning(sweep_persistent=chained)
        s.init_flowfield()
        got.append(run(s, 4))
        s.close()
    assert all(np.array_equal(a, b) for a, b in zip(*got))
    assert np.isfinite(got[0][0]).all()


def test_natural_order_is_chained_by_default_and_a_batch_runs_it():
    cases = [case("bump_small"), case("plate2d")]
    one = [Solver(m, p) for m, p in cases]
    assert [s.tuning()["sweep_persistent"] for s in one] == [1, 1]
    assert Solver(*case("bump_colour")).tuning()["sweep_persistent"] == 0
    for s in one:
        s.init_flowfield()
    many = [Solver(m, p) for m, p in cases]
    for s in many:
        s.init_flowfield()
    b = Batch(many)
    b.step(5)
    for s, t in zip(one, many):
        s.step(5)
        assert np.array_equal(s.state(), t.state())
    b.close()
