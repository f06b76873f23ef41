"""The incompressible solver's GMRES kernels at the sizes where their tiling
can go wrong: systems smaller than one 256-row chunk, of a few chunks with a
ragged last one (an odd number of rows), of two chunks a block, solves that
converge before the products are split over several blocks, that pass many
rounds of it, and that run out of Krylov vectors (500).  Against the CPU
restatement, held as in test_gpu_ins.py: the same iteration counts, fields to
1e-9 of their magnitude (operations in the reference's order but for the
blocked inner products)."""
import numpy as np
import pytest

from oneflow_b200 import meshgen, params as P
from oneflow_b200.solver import Incompressible
from oracle_lib import InsOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,triangles", [(6, False), (17, False), (33, True), (90, False)])
def test_solves_match_the_restatement(n, triangles):
    mesh = meshgen.lid_cavity_2d(n, jitter=0.1, triangles=triangles)
    prm = P.defaults(vismodel=1, reynolds=1000.0, mach_ref=0.1)
    wall = meshgen.lid_velocity(mesh)
    g, o = Incompressible(mesh, prm, wall), InsOracle(mesh, prm, wall)
    g.update_residuals()
    o.run(1)
    sg, so = g.stats(), o.stats()
    assert list(sg["gmres_iters"]) == list(so["gmres_iters"])
    for k in ("pp", "uc", "vc"):
        a, b = g.field(k), o.field(k)
        assert np.abs(a - b).max() <= 1e-9 * max(np.abs(b).max(), 1e-300), k


def test_a_second_chunk_round_repeats_itself():
    # 350 x 350: 486 chunks for 444 resident blocks; no restatement of that
    # size, but the solve must be the same run to run and reduce its residual
    mesh = meshgen.lid_cavity_2d(350, jitter=0.1)
    prm = P.defaults(vismodel=1, reynolds=1000.0, mach_ref=0.1)
    out = []
    for _ in range(2):
        g = Incompressible(mesh, prm, meshgen.lid_velocity(mesh))
        g.update_residuals()
        out.append((g.q(), g.stats()))
        g.close()
    assert np.array_equal(out[0][0], out[1][0])
    s = out[0][1]
    assert s["gmres_iters"][0] < 60 and s["gmres_res"][0] < 1e-7   # the momentum solve converged
    assert np.isfinite(out[0][0]).all()
