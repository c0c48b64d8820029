"""Reading and writing multigrid planes (stored row by row with a pitch, given
column by column): what is written comes back bit for bit, on planes that end
inside a 32 x 32 tile and on levels of one row, and the agar view is the
solution's rows 1 .. box_z_agar without its last column."""
import numpy as np
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony


@pytest.mark.gpu
@pytest.mark.parametrize("box_x,rows,levels", [(256, 32, 2), (224, 31, 2), (288, 65, 1), (992, 2, 3)])
def test_planes_round_trip(gpu, box_x, rows, levels):
    p = params.parse_parameters(params.shipped_input_text("small"))
    p.box_x, p.box_y, p.box_z, p.box_z_agar, p.max_levels_mg, p.max_cells, p.mg_levels = box_x, 1, 20, rows, levels, 16, 6
    col = Colony(params.finalize(p))
    rng = np.random.default_rng(box_x)
    names = ["MG_%s_%s" % (k, s) for k in ("SOL", "RES", "ERR") for s in ("CARBON", "OXYGEN", "ACETATE")]
    put = {}
    for name in names:
        for l in range(p.mg_levels):
            put[name, l] = rng.standard_normal(col.field(name, l).size)
            col.set_field(name, put[name, l], l)
    for (name, l), v in put.items():
        assert np.array_equal(col.field(name, l), v), (name, l)
    for s in ("CARBON", "OXYGEN", "ACETATE"):
        for l in range(levels):
            sol = put["MG_SOL_" + s, l].reshape(box_x + 1, rows + 1)
            assert np.array_equal(col.field("AGARF_" + s, l).reshape(box_x, rows), sol[:box_x, 1:])
    col.close()
