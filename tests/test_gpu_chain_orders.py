"""The chained LU-SGS sweeps in a cluster of blocks on level structures that try
their orders: levels of one cell between levels that occupy every warp, and
neighbours that the ring no longer holds, read a few levels after they were
written, and levels wider than the ring, whose cells share its slots.  Against one launch per level: the same bits."""
import numpy as np
import pytest

from oneflow_b200 import meshgen, params as P
from oneflow_b200.meshio import Mesh
from oneflow_b200.solver import TURB_SOLVER, Solver
from oneflow_b200.walldist import plate_wall_distance

pytestmark = pytest.mark.gpu


def ladder(width, rows):
    """Rows of ``width`` quadrilaterals, each row under two cells as long as the row.
    Numbered row by row: every other quadrilateral, then the two long cells; the other
    quadrilaterals last.  Levels of width / 2, one and width / 2 + 1 cells in turn."""
    xs = np.linspace(0.0, 3.0, width + 1)
    h = 1.0 / (3 * rows)
    x, y, fine, ends = [], [], [], []
    for r in range(rows):
        for k in (0, 1):
            fine.append(len(x) + np.arange(width + 1))
            x += list(xs); y += [(3 * r + k) * h] * (width + 1)
        ends.append((len(x), len(x) + 1))
        x += [0.0, 3.0]; y += [(3 * r + 2) * h] * 2
    fine.append(len(x) + np.arange(width + 1))
    x += list(xs); y += [1.0] * (width + 1)
    cells, last = [], []
    for r in range(rows):
        lo, hi, nxt, (a, b) = fine[2 * r], fine[2 * r + 1], fine[2 * r + 2], ends[r]
        for i in range(width):
            (cells if i % 2 == 0 else last).append((lo[i], lo[i + 1], hi[i + 1], hi[i]))
        cells.append(tuple(hi) + (b, a))
        cells.append((a, b) + tuple(nxt[::-1]))
    x, y = np.array(x), np.array(y)
    bc = lambda a, b: meshgen.FAR if x[a] == x[b] else meshgen.SOLID   # noqa: E731
    nodes, lc, rc, nb, bct = meshgen._faces_from_cells_2d(cells + last, bc)
    return Mesh(2, x, y, np.zeros_like(x), np.full(len(lc), 2, np.int32), nodes.ravel().astype(np.int32),
                lc.astype(np.int32), rc.astype(np.int32), len(cells) + len(last), nb, bct)


def shuffled(m, seed):
    return m.renumber_cells(np.random.default_rng(seed).permutation(m.n_cells))


def both(m, prm, steps=4):
    got = []
    for chained in (0, 1):
        s = Solver(m, prm)
        s.set_tuning(sweep_persistent=chained)
        s.init_flowfield()
        s.step(steps)
        got.append([s.state(), s.res_history()] + ([s.state(TURB_SOLVER)] if prm.vismodel >= 3 else []))
        s.close()
    assert np.isfinite(got[0][0]).all()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("width,rows,precision", [(1100, 7, 1), (1550, 5, 0)])   # clusters of 4 and 8 blocks
def test_levels_of_one_cell_between_wide_ones(width, rows, precision):
    both(ladder(width, rows), P.euler_bump(precision=precision))


@pytest.mark.parametrize("precision", [0, 1])
def test_neighbours_beyond_the_ring_a_few_levels_on(precision):
    both(shuffled(meshgen.bump_channel(60, 40), 20), P.euler_bump(precision=precision, ilim=2, vencat_coef=0.05))


@pytest.mark.parametrize("name", ["bump_4k", "bump_7k", "bump_mixed", "ladder", "plate3d", "plate3d_fp64"])
def test_levels_wider_than_the_ring(name):
    """widest levels of 4,200 to 12,400 cells, narrower ones after them"""
    if name == "ladder":   # its upper sweep begins with one level of half the quadrilaterals
        return both(ladder(3100, 8), P.euler_bump())
    if name.startswith("bump"):
        ni, nj, precision = {"bump_4k": (110, 70, 0), "bump_7k": (140, 100, 0), "bump_mixed": (140, 100, 1)}[name]
        return both(shuffled(meshgen.bump_channel(ni, nj), 21),
                    P.euler_bump(precision=precision, ilim=2, vencat_coef=0.05))
    m = meshgen.flat_plate_tets(26, 16, 10)
    m.wall_dist = plate_wall_distance(m)
    both(shuffled(m, 1), P.rans_plate(precision=0 if name == "plate3d_fp64" else 1, sweep_order=0))
