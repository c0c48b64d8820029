"""Several colony sweeps in one launch against one launch a sweep: the same
operations in the same order, so every field is equal bit for bit.  Setting
the bounding box through bcg_set_bbox, to what it was, selects the single
sweeps (a box that is not the deposition's).  Sizes around a tile's edges: 4, 8 and
16 columns, 35 and 38 rows, the launches' 4 sweeps in pairs."""
import numpy as np
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony, packed_colony

FIELDS = ("ENV_CARBON", "ENV_WASTE", "ENV_OXYGEN", "ENV_ACETATE", "ENV_GROWTH1", "ENV_PH", "ENV_BUFFER", "ENV_GR_CAR_AER",
          "OLDENV_CARBON", "OLDENV_WASTE", "OLDENV_OXYGEN", "OLDENV_ACETATE")
WALLS = ("WALLF_CARBON", "WALLF_WASTE", "WALLF_OXYGEN", "WALLF_ACETATE",
         "OLDWALLF_CARBON", "OLDWALLF_WASTE", "OLDWALLF_OXYGEN", "OLDWALLF_ACETATE")


def colony(n, width, height, box_x, box_z, levels):
    p = params.parse_parameters(params.shipped_input_text("small"))
    p.box_x, p.box_y, p.box_z, p.box_z_agar, p.max_levels_mg, p.max_cells = box_x, 1, box_z, 16, levels, n + 64
    p.mg_levels = 5
    p = params.finalize(p)
    col = Colony(p, packed_colony(n, width, height, seed=n))
    col.initial_density()
    return col


def state(col):
    out = [col.field(f) for f in FIELDS]
    return out + [col.field(w, l) for w in WALLS for l in range(col.params.max_levels_mg)]


# width and height (um) of the dome; a box is 4 um, the field box 5 boxes more
SHAPES = {
    "narrow": (60, 15.0, 30.0, 64, 24, 2),
    "wide": (900, 420.0, 14.0, 192, 20, 3),
    "one level": (500, 200.0, 16.0, 160, 24, 1),
    "rows 37": (1500, 60.0, 125.0, 128, 48, 2),      # the box's top near the one-tile limit
    "rows 38": (1500, 60.0, 129.0, 128, 48, 2),
    "rows 39": (1500, 60.0, 133.0, 128, 56, 2),
    "two tiles": (3000, 90.0, 200.0, 128, 72, 2),
    "three tiles": (4000, 90.0, 300.0, 128, 100, 2),
    "tiles of 8": (6500, 2900.0, 14.0, 800, 20, 2),
    "tiles of 16": (13000, 5800.0, 14.0, 1536, 20, 3),
    "at the edge": (600, 200.0, 20.0, 76, 24, 2),    # tiles would reach the grid's sides
}


@pytest.mark.gpu
@pytest.mark.parametrize("shape", list(SHAPES))
def test_blocked_sweeps_equal_single(gpu, shape):
    a, b = colony(*SHAPES[shape]), colony(*SHAPES[shape])
    b.set_bbox(*b.bbox())
    for sweeps, count0 in ((8, 0), (10, 0), (19, 1), (7, 0), (26, 3), (1, 0), (0, 0)):
        la, lb = a.kernel_launches(), b.kernel_launches()
        a.colony_sweeps(sweeps, count0)
        b.colony_sweeps(sweeps, count0)
        if sweeps == 26 and shape != "at the edge":
            assert a.kernel_launches() - la < b.kernel_launches() - lb     # 6 blocked + types + 2
        for x, y in zip(state(a), state(b)):
            assert np.array_equal(x, y), (shape, sweeps, count0)
    # whole updates, whose units replay as graphs; the box changes hands between
    a.nutrient_update(3, 20)
    b.nutrient_update(3, 20)
    a.set_bbox(*a.bbox())
    a.nutrient_update(2, 20)
    b.nutrient_update(2, 20)
    for x, y in zip(state(a), state(b)):
        assert np.array_equal(x, y), shape
    a.close()
    b.close()
