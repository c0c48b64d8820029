"""The register-tiled smoother and the one-launch coarsest levels (relax mode
3's small levels) against the form that relaxes one column a thread, row by
row (relax mode 0): whole solves, so that descent, coarsest level and ascent
all enter.  The two differ only in how a column's recurrence is rounded: 1e-12
of the largest solution value, as the solves against the oracle are held to."""
import ctypes

import numpy as np
import pytest

from baccolonygrowth_b200 import _abi, params
from baccolonygrowth_b200.colony import Colony, synth_colony

SPECIES = ("CARBON", "OXYGEN", "ACETATE")


def problem(box_x, rows, levels, **kw):
    p = params.parse_parameters(params.shipped_input_text("small"))
    p.box_x, p.box_y, p.box_z, p.box_z_agar, p.max_levels_mg, p.max_cells = box_x, 1, 24, rows, levels, 512
    for k, v in kw.items():
        setattr(p, k, v)
    return params.finalize(p)


def colony(p, mode):
    w, h = params.dome_size(200, 1.0 / 10.0)
    col = Colony(p, synth_colony(200, w, h, seed=5))
    _abi.check(col.lib.bcg_set_relax_mode(col.h, mode), "mode")
    col.update_density()
    col.deplete_wall()
    return col


def solutions(col):
    return [col.field("MG_SOL_" + s, l) for s in SPECIES for l in range(col.params.max_levels_mg)]


@pytest.mark.gpu
@pytest.mark.parametrize("box_x,rows,levels,kw", [
    (128, 2, 1, {"mg_levels": 6}),            # levels of one row and of none inside
    (128, 16, 2, {}),
    (160, 17, 2, {}),                         # odd column counts on the coarse levels
    (224, 35, 3, {}),                         # 36 rows: four whole chunks
    (256, 32, 2, {"mg_mu1": 1}),
    (256, 36, 2, {"mg_mu1": 2}),              # one row into a fifth chunk
    (256, 128, 2, {"mg_mu1": 4}),             # two launches a smoothing
    (416, 143, 3, {}),                        # the most rows one block takes, less one
    (416, 144, 3, {}),                        # ... and one more: two segments
    (448, 300, 2, {}),                        # four segments
    (992, 40, 5, {}),                         # coarse levels beside rows without padding
    (1024, 64, 3, {"mg_mu2": 7}),             # the coarsest level stops before its fixed point
    (4608, 24, 3, {"mg_levels": 6}),          # a coarsest level of many columns
    (512, 64, 8, {}),                         # every level composite
])
def test_solve_equals_column_form(gpu, box_x, rows, levels, kw):
    p = problem(box_x, rows, levels, **kw)
    a, b = colony(p, 3), colony(p, 0)
    for k in range(3):
        a.mg_solve()
        b.mg_solve()
    for x, y in zip(solutions(a), solutions(b)):
        assert np.abs(x - y).max() <= 1e-12 * max(np.abs(y).max(), 1e-300)
    a.close()
    b.close()
