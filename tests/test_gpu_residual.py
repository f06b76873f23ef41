"""The FP64 residual pass on either side of its dispatch (four lanes a cell on
small meshes, a thread a cell above; the TEST / NEW1 / NEW2 viscous schemes
always the latter) against the CPU oracle: cells at the edges of warps, blocks
and clusters, more than four faces a cell, and the norms' block sums."""
import numpy as np
import pytest

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import LUSGS_SEQUENCE, Solver
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 5), (4, 4), (13, 5), (8, 8), (43, 3), (64, 32), (75, 60), (90, 51)]


def cases():
    for n in SIZES:
        yield f"bump_{n[0]}x{n[1]}", lambda n=n: (meshgen.bump_channel(*n), P.euler_bump(ilim=2, vencat_coef=0.05))
    yield "hexes", lambda: (meshgen.bump_box_hexes(5, 4, 3), P.euler_bump(dimension=3))
    yield "hybrid", lambda: (meshgen.bump_box_mixed(8, 6, 4), P.euler_bump(dimension=3, ilim=1))
    for n in ((7, 5), (24, 16), (100, 90), (91, 100)):
        yield f"plate_{n[0]}x{n[1]}", lambda n=n: (
            meshgen.plate_2d(*n), P.defaults(ischeme=12, ilim=0, mach_ref=0.2, reynolds=1e5, vismodel=1))


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-30))


@pytest.mark.parametrize("name,make", list(cases()), ids=[n for n, _ in cases()])
def test_residual_pass(name, make):
    m, prm = make()
    o, g = Oracle(m, prm), Solver(m, prm)
    o.init()
    g.init_flowfield()
    N = m.n_cells
    for it in range(2):
        o.task("NEXT_STEP")
        g.set_outer_step(it + 1)
        for t in LUSGS_SEQUENCE:
            o.task(t)
            g.task(t)
            if t == "CALC_TIME_STEP":
                for f in ("timestep", "invsr", "vissr"):
                    assert rel(g.field(f)[:N], o.field(f)[:N]) < 1e-12, (it, f)
            if t == "UPDATE_RESIDUALS":
                # round-off of the per-cell sums: as the task-by-task parity tests
                r = g.field("res").reshape(5, -1)[:, :N]
                assert rel(r, o.field("res").reshape(5, -1)[:, :N]) < 1e-11, it
                # the norms' own sums: N positive terms in FP64, then a root
                want = np.sqrt((r.astype(np.longdouble) ** 2).sum(axis=1) / N).astype(np.float64)
                assert np.allclose(g.residual_norms(), want, rtol=N * 2.3e-16 + 1e-14, atol=0), it
