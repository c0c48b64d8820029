"""One lane a cell stages its neighbours' records or gathers them, by colony
size and precision: the same arithmetic in the same order, so a colony one
cell above the line moves like the same colony without that cell (which
stands alone at the grid's side), bit for bit."""
import numpy as np
import pytest

from baccolonygrowth_b200 import _abi, params
from baccolonygrowth_b200.colony import Colony, Rng, packed_colony


@pytest.mark.gpu
@pytest.mark.parametrize("n,bits", [(100000, 32), (200000, 64)])
def test_staged_equals_gathered(gpu, n, bits):
    p = params.ensemble_member(n)
    p.box_x += 16
    p.max_cells = n + 8
    params.finalize(p)
    cells = packed_colony(n + 1, *params.dome_size(n, 1.0 / 20.0, 0.9))
    cells["ldiv"] = 100.0
    for q, dx in (("p", -1.0), ("q", 1.0)):
        cells[q][n] = ((-(p.box_x // 2) + 3) * p.box_length + dx, 0.0, 0.6)
    cells["length"][n] = 2.0
    assert np.abs(cells["p"][:n, 0] - cells["p"][n, 0]).min() > 20.0
    out, fields = [], None
    for m in (n, n + 1):
        col = Colony(p, cells[:m])
        if fields is None:
            col.update_density()
            fields = {f: col.field(f) for f in ("HEIGHT", "NORMAL_X", "NORMAL_Z", "WALL")}
        for f, v in fields.items():
            col.set_field(f, v)
        col.set_field("ENV_GROWTH1", np.full(p.box_x * p.box_z, 0.9))
        col.rebuild_neighbours()
        col.set_pair_precision(bits)
        assert _abi.load().bcg_set_force_group(col.h, 1) == 0
        for k in range(3):
            assert len(col.step(p.dt, k * p.dt, Rng(1))) == 0
        out.append(col.cells()[:n])
        col.close()
    assert out[0].tobytes() == out[1].tobytes()
    assert np.abs(out[0]["velocity"]).max() > 0
