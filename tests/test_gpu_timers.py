"""The launches that a timer reports are those of its calls, whatever form their
kernels take (a scan in one block or in three launches, by the number of boxes)."""
import numpy as np
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony, Rng, packed_colony


@pytest.mark.gpu
@pytest.mark.parametrize("box_x,box_z", [(256, 128), (256, 129)])
@pytest.mark.parametrize("dividing", [0, 5])
def test_timer_launches(gpu, box_x, box_z, dividing):
    p = params.ensemble_member(600)
    p.box_x, p.box_z = box_x, box_z
    params.finalize(p)
    cells = packed_colony(600, *params.dome_size(600, 1.0 / 20.0, 0.9))
    cells["ldiv"] = 10.0
    cells["ldiv"][:dividing] = cells["length"][:dividing]
    col = Colony(p, cells)
    col.set_field("ENV_GROWTH1", np.full(p.box_x * p.box_z, 0.9))
    col.enable_timers()
    rng = Rng(5)
    for name, call in (("DENSITY", col.update_density), ("DENSITY", col.update_height), ("NEIGHBOURS", col.rebuild_neighbours),
                       ("MOVE_GROW", lambda: col.move_grow(p.dt)),
                       ("DIVIDE", lambda: col.divide(rng.frand(9 * dividing), 0.0)),
                       ("MG_SOLVE", col.mg_solve), ("MG_SOLVE", col.mg_solve), ("SWEEPS", lambda: col.colony_sweeps(20)),
                       ("SWEEPS", lambda: col.nutrient_update(3, 20))):
        l0, t0 = col.kernel_launches(), col.timer(name)[1]
        call()
        assert col.timer(name)[1] - t0 == col.kernel_launches() - l0, name
    col.close()
