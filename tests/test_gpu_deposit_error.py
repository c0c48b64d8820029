"""A deposition that ends with an error leaves no bounding box for the blocked
sweeps to go by: the next sweeps run one a launch, as after bcg_set_bbox, until a
deposition has ended well."""
import pytest

from baccolonygrowth_b200 import _abi, params
from baccolonygrowth_b200.colony import Colony, packed_colony


def launches(col, sweeps):
    l0 = col.kernel_launches()
    col.colony_sweeps(sweeps)
    return col.kernel_launches() - l0


@pytest.mark.gpu
def test_sweeps_after_failed_deposition(gpu):
    p = params.parse_parameters(params.shipped_input_text("small"))
    p.box_x, p.box_y, p.box_z, p.box_z_agar, p.max_levels_mg, p.max_cells, p.mg_levels = 128, 1, 24, 16, 2, 512, 5
    p = params.finalize(p)
    p.max_cells_per_box = 12
    cells = packed_colony(300, 120.0, 16.0, seed=3)
    fits, crowded = cells[:20], cells.copy()
    crowded["p"][:20], crowded["q"][:20] = cells["p"][0], cells["q"][0]     # twenty cells in one box
    col = Colony(p, fits)
    col.update_density()
    assert launches(col, 26) < 26
    col.upload(crowded)
    with pytest.raises(_abi.BcgError) as e:
        col.update_density()
    assert e.value.code == _abi.E_BOX_OVERFLOW
    assert launches(col, 26) == 26
    col.upload(fits)
    col.update_density()
    assert launches(col, 26) < 26
    col.close()
