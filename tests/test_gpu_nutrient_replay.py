"""A nutrient update whose units replay captured graphs against one that
captures them anew (changing the smoother form and back drops the graphs):
the same kernels on the same values, so all of it is equal bit for bit, also
what the library works out only when it is read (level 0's Res after a solve)
and the second agar buffer that the legacy solver takes up after a solve."""
import numpy as np
import pytest

from baccolonygrowth_b200 import params
from baccolonygrowth_b200.colony import Colony, workload_colony

pytestmark = pytest.mark.gpu
SPECIES = ("CARBON", "OXYGEN", "ACETATE")


def pair():
    out = []
    for _ in range(2):
        col = Colony(params.workload_params("small_4k"), workload_colony("small_4k", n=1024))
        col.update_density()
        col.deplete_wall()
        out.append(col)
    return out


def recapture(col):
    for mode in (2, 3):
        assert col.lib.bcg_set_relax_mode(col.h, mode) == 0


def update(a, b, units=2):
    """`a` replays, `b` captures."""
    recapture(b)
    a.nutrient_update(units)
    b.nutrient_update(units)


def equal(a, b, names):
    for name in names:
        for l in range(a.params.max_levels_mg):
            assert np.array_equal(a.field(name, l), b.field(name, l)), (name, l)


@pytest.mark.parametrize("between", ["density", "read", "none"])
def test_res_after_replay(gpu, between):
    a, b = pair()
    update(a, b)
    for _ in range(2):
        for col in (a, b):
            if between == "density":
                col.update_density()
            elif between == "read":
                col.field("MG_SOL_CARBON", 0)
        update(a, b)
    equal(a, b, ["MG_%s_%s" % (k, s) for k in ("RES", "ERR", "SOL") for s in SPECIES])
    assert np.abs(a.field("MG_RES_CARBON", 0)).max() > 0
    a.close(); b.close()


@pytest.mark.parametrize("solve", ["update", "mg_solve"])
def test_res_is_of_the_field_the_solve_saw(gpu, solve):
    """Level 0's Res read before a deposition of other cells and after it, and
    after two."""
    out = []
    for depositions in (0, 1, 2):
        col, other = pair()
        other.close()
        for k in range(3):
            col.nutrient_update(2) if solve == "update" else col.mg_solve()
            if k < 2:
                col.update_density()
        for d in range(depositions):
            cells = workload_colony("small_4k", n=1024)
            cells["p"][:, 0] += 40.0 * (d + 1)
            cells["q"][:, 0] += 40.0 * (d + 1)
            before = col.field("INSIDE")
            col.upload(cells)
            col.update_density()
            assert not np.array_equal(before, col.field("INSIDE"))
        out.append([col.field("MG_RES_" + s, 0) for s in SPECIES])
        col.close()
    for o in out[1:]:
        for x, y in zip(out[0], o):
            assert np.abs(x).max() > 0 and np.array_equal(x, y)


def test_res_is_of_the_field_before_it_is_set(gpu):
    """insideColonyDen that a caller sets after a solve does not reach the Res
    that the solve left."""
    a, b = pair()
    for col in (a, b):
        col.mg_solve()
    want = [a.field("MG_RES_" + s, 0) for s in SPECIES]
    b.set_field("INSIDE", 1.0 - b.field("INSIDE"))
    for s, w in zip(SPECIES, want):
        assert np.array_equal(b.field("MG_RES_" + s, 0), w), s
    a.close(); b.close()


def test_legacy_after_replay(gpu):
    a, b = pair()
    update(a, b)
    for _ in range(2):
        for col in (a, b):
            col.legacy_env_update(3)
        update(a, b)
    for col in (a, b):
        col.legacy_env_update(3)
    equal(a, b, ["AGARF_" + s for s in SPECIES] + ["%sWALLF_%s" % (o, s) for o in ("", "OLD") for s in SPECIES])
    a.close(); b.close()


def test_replay_after_write(gpu):
    """Err and Res that a caller wrote are not taken for the zeros a solve
    leaves."""
    a, b = pair()
    update(a, b)
    err = np.random.default_rng(1).standard_normal(a.field("MG_ERR_CARBON", 0).size)
    for col in (a, b):
        col.set_field("MG_ERR_CARBON", err, 0)
    update(a, b)
    equal(a, b, ["MG_SOL_" + s for s in SPECIES])
    a.close(); b.close()
