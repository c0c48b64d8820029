"""The mechanics and deposition kernels at the edges of their dispatch, against
the C restatement in oracle/: the number of lanes a cell by colony size, the
one-block scan, the candidate list's window, the division draws' two routes,
and the per-column deposition.

Bars as in test_gpu_mechanics.py and test_gpu_fields.py: neighbour sets,
division events, flags and heights exact; cells within 1e-10 relative,
densities within 1e-12.
"""
import numpy as np
import pytest

from baccolonygrowth_b200 import _abi, params
from baccolonygrowth_b200.colony import Colony, Rng, packed_colony

import checkers as ck
from test_gpu_fields import bbox_mask, close
from test_gpu_mechanics import assert_cells_close, nbr_sets

F = _abi.FIELDS
pytestmark = pytest.mark.gpu


def make(n, mutate=None, seed=77, box_x=None, box_z=None, phi=0.9):
    p = params.ensemble_member(n)
    p.box_x, p.box_z = box_x or p.box_x, box_z or p.box_z
    params.finalize(p)
    w, h = params.dome_size(n, 1.0 / 20.0, phi)
    cells = packed_colony(n, w, h)
    if mutate is not None:
        mutate(cells)
    orc = ck.Oracle(p, seed=seed)
    orc.load(cells)
    orc.update_density()
    orc.set_field(F["ENV_GROWTH1"], np.full(p.box_x * p.box_z, 0.9))
    orc.rebuild()
    col = Colony(p, cells)
    for f in ("HEIGHT", "NORMAL_X", "NORMAL_Z", "WALL", "ENV_GROWTH1"):
        col.set_field(f, orc.field(F[f]))
    col.rebuild_neighbours()
    rng = Rng(seed)
    for _ in range(p.box_x * p.box_y):   # the wall draws
        rng.next()
    return p, orc, col, rng


def step_both(p, orc, col, rng):
    _, _, lin_o = orc.step(p.dt, 0.0)
    lin = col.step(p.dt, 0.0, rng)
    assert np.array_equal(lin, lin_o)
    assert_cells_close(orc.cells(), col.cells())
    assert nbr_sets(orc.neighbours()) == nbr_sets(col.neighbours())
    return len(lin)


# one wave of 75776 lanes holds 8, 4 and 2 lanes for 9472, 18944 and 37888 cells
@pytest.mark.parametrize("n", [33, 9472, 9473, 18945, 37889])
def test_default_lanes(gpu, n):
    step_both(*make(n))


@pytest.mark.parametrize("group", [1, 16])
@pytest.mark.parametrize("n", [31, 129, 4097])
def test_lanes_on_partial_warps(gpu, n, group):
    p, orc, col, rng = make(n)
    assert _abi.load().bcg_set_force_group(col.h, group) == 0
    step_both(p, orc, col, rng)


def test_one_cell(gpu):
    """A lone cell's wall torques cancel, so its angular velocity is rounding
    (nothing to compare with the oracle's): all lane counts do the same
    arithmetic on it and agree in every bit."""
    out = []
    for group in (1, 2, 16):
        p, _, col, rng = make(1)
        assert _abi.load().bcg_set_force_group(col.h, group) == 0
        col.step(p.dt, 0.0, rng)
        out.append(col.cells())
    assert out[0].tobytes() == out[1].tobytes() == out[2].tobytes()


# 256 x 128 boxes are the last that one block scans
@pytest.mark.parametrize("box_z", [16, 127, 128, 129])
def test_scan_sizes(gpu, box_z):
    p, orc, col, rng = make(1025, box_x=256, box_z=box_z)
    assert nbr_sets(orc.neighbours()) == nbr_sets(col.neighbours())
    step_both(p, orc, col, rng)


def squeeze(f):
    def mutate(cells):
        for q in ("p", "q"):
            cells[q] *= f      # shorter cells, closer together: more of them in a box
        cells["length"] *= f
    return mutate


# a lane group's candidate list holds 64: fewer, and several windows of it
@pytest.mark.parametrize("f", [1.0, 0.7, 0.5])
def test_candidate_windows(gpu, f):
    p, orc, col, rng = make(2000, mutate=squeeze(f))
    assert nbr_sets(orc.neighbours()) == nbr_sets(col.neighbours())


# up to 64 divisions read their draws where the host wrote them
@pytest.mark.parametrize("count", [1, 63, 64, 65])
def test_division_counts(gpu, count):
    def mutate(cells):
        cells["ldiv"] = 10.0
        pick = np.random.default_rng(3).permutation(len(cells))[:count]
        cells["ldiv"][pick] = cells["length"][pick]
    assert step_both(*make(3000, mutate=mutate)) == count


@pytest.mark.parametrize("n,box_z", [(1, None), (700, 33), (20000, None), (60000, 131)])
def test_deposition_sizes(gpu, n, box_z):
    p, orc, col, _ = make(n, box_z=box_z, phi=0.45)
    col.update_density()
    orc.update_density()
    assert orc.bbox() == col.bbox()
    for f in ("INSIDE", "HEIGHT"):
        assert np.array_equal(orc.field(F[f]), col.field(f)), f
    m = bbox_mask(p, orc.bbox())
    assert close(orc.field(F["ROUGH_DENSITY"]), col.field("ROUGH_DENSITY"), mask=m) <= 1e-12
    orc.update_height()
    col.update_height()
    assert np.array_equal(orc.field(F["HEIGHT"]), col.field("HEIGHT"))
