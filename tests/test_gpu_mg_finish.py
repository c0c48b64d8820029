"""The passes that end a solve (update, nesting, boundary rewrite, zeroing, wall
rows: two launches over all levels) against the C restatement in oracle/, by the
number of composite levels: one (nothing nests), three and five (a point is
nested several times).  Bars as test_gpu_fields.py's test_mg_solve."""
import numpy as np
import pytest

from baccolonygrowth_b200 import _abi, params
from baccolonygrowth_b200.colony import Colony, synth_colony

import checkers as ck
from test_gpu_fields import TOL, close, deplete, wall_mask
from test_gpu_mg_tile import colony, problem, solutions

F = _abi.FIELDS
SPECIES = ("CARBON", "OXYGEN", "ACETATE")


@pytest.mark.gpu
@pytest.mark.parametrize("box_x,rows,levels", [(256, 16, 1), (224, 36, 3), (992, 40, 5)])
def test_solve_end_against_oracle(gpu, box_x, rows, levels):
    p = problem(box_x, rows, levels)
    w, h = params.dome_size(200, 1.0 / 10.0)
    cells = synth_colony(200, w, h, seed=5)
    orc = ck.Oracle(p, seed=12345)
    orc.load(cells)
    col = Colony(p, cells)
    col.set_field("WALL", orc.field(F["WALL"]))
    orc.update_density()
    col.update_density()
    deplete(p, orc, col)
    for _ in range(2):
        orc.mg_solve(2, p.mg_dt)
        col.mg_solve(2)
    for l in range(p.mg_levels):
        for sp in SPECIES:
            for kind in ("SOL", "RES", "ERR"):
                f = "MG_%s_%s" % (kind, sp)
                a, b = orc.field(F[f], l), col.field(f, l)
                if kind == "SOL":
                    assert close(a, b) <= TOL, (f, l)
                else:
                    assert np.abs(a - b).max() <= TOL * max(1.0, np.abs(a).max()), (f, l)
    for l in range(p.max_levels_mg):
        for sp in SPECIES:
            f = "WALLF_" + sp
            assert close(orc.field(F[f], l), col.field(f, l), mask=wall_mask(p, l)) <= TOL, (f, l)


# the cluster form of the coarsest level stops at its fixed point: sweeps that
# end before a row's wavefront has, before the fixed point, and long after it
@pytest.mark.gpu
@pytest.mark.parametrize("mu2", [1, 2, 9, 40, 300])
def test_coarsest_level_stops_at_fixed_point(gpu, mu2):
    p = problem(4608, 24, 3, mg_levels=6, mg_mu2=mu2)
    a, b = colony(p, 3), colony(p, 0)
    for _ in range(2):
        a.mg_solve()
        b.mg_solve()
    for x, y in zip(solutions(a), solutions(b)):
        assert np.abs(x - y).max() <= 1e-12 * max(np.abs(y).max(), 1e-300)


# blocks of 16 rows, eight loaded together; 37 rows of points.  Without sweeps the
# correction stays zero, so the relaxation's defect is Res itself and the ratio 1
# up to the rounding of c R (cf + 2) / cf; a row that were left out would give 0.
@pytest.mark.gpu
@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("k", [1, 7, 8, 9, 14, 15, 16, 17, 24, 31, 32, 33, 35])
def test_defect_sees_every_row(gpu, k, precision):
    p = problem(256, 36, 2, mg_mu1=0, mg_mu2=0)
    col = Colony(p, synth_colony(200, *params.dome_size(200, 1.0 / 10.0), seed=5))
    for l in range(2):
        n = len(col.field("MG_SOL_CARBON", l))
        sol = np.full((n // 37, 37), 8.0)
        if l == 0:
            sol[101, k] = 7.0
        col.set_field("MG_SOL_CARBON", sol.reshape(-1), l)
    it, rel = col.mg_solve_tol(1e-300, precision, 1)
    assert it == 1 and abs(rel - 1.0) <= 1e-14, (it, rel)
    col.close()
