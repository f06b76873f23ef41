"""Device memory that only buys speed (the chained sweeps' schedules, the second
set of gradient records of the overlapped SA iteration) is not taken on a device
that is more than half full: a solve that fits without it fits, and gives the
same bits."""
import numpy as np
import pytest
import torch

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import TURB_SOLVER, Solver
from oneflow_b200.walldist import plate_wall_distance

pytestmark = pytest.mark.gpu


def case(name):
    if name == "chain":   # natural order: about 60,000 edges a sweep at 140 bytes each, two schedules and a scratch
        return meshgen.bump_channel(230, 90), P.euler_bump(precision=0, sweep_order=0), 10 << 20
    m = meshgen.flat_plate_tets(60, 40, 10)
    m.wall_dist = plate_wall_distance(m)
    prm = P.rans_plate(precision=0, sweep_order=1, igrad=0, venkat_kh3=0, vencat_coef=0.0001)
    return m, prm, m.n_cells * 24 * 8   # 24 FP64 values a cell


def fill(leave):
    """Everything of the device but ``leave`` bytes."""
    torch.cuda.empty_cache()
    return torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")


def solve(m, prm):
    before = torch.cuda.mem_get_info()[0]
    s = Solver(m, prm)
    taken = before - torch.cuda.mem_get_info()[0]
    s.init_flowfield()
    s.step(3)
    out = [s.state()] + ([s.state(TURB_SOLVER)] if prm.vismodel >= 3 else [])
    s.close()
    return taken, out


@pytest.mark.parametrize("name", ["chain", "overlap"])
def test_a_full_device_keeps_to_what_a_solve_needs(name):
    m, prm, extra = case(name)
    solve(m, prm)   # kernels loaded
    most, want = solve(m, prm)
    total = torch.cuda.mem_get_info()[1]
    held = fill(int(0.4 * total))
    least, got = solve(m, prm)
    assert most - least >= 0.8 * extra
    assert all(np.array_equal(a, b) for a, b in zip(want, got))
    del held
    held = fill(least + (96 << 20))   # and what a few steps need
    assert all(np.array_equal(a, b) for a, b in zip(want, solve(m, prm)[1]))
    del held
    torch.cuda.empty_cache()
