"""Rows of the blocked colony sweeps' tiles: every row of the bounding box has
one owner (two blocks of a launch would write it otherwise), and the number of
tile rows is the one that the launch's tile width is chosen by.  The rule is
plain C++ (csrc/sweep_rows.h), compiled here with the host compiler; on the GPU,
boxes whose top lies around the bottom tile's last rows against single sweeps."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "baccolonygrowth_b200", "csrc")

PROBE = r"""
#include <cstdio>
#include "sweep_rows.h"
int main()
{
    /* a block of tile row zt runs if sw_runs says so and then stores its rows up to maxz */
    for (int maxz = 0; maxz < 400; maxz++) {
        const int rows = sw_tile_rows(maxz);
        printf("%d %d", maxz, rows);
        for (int z = 0; z <= maxz; z++) {
            int owners = 0;
            for (int zt = 0; zt < 20; zt++) owners += sw_runs(zt, maxz) && z >= sw_first(zt) && z < sw_end(zt, maxz);
            if (owners != 1) printf(" row %d has %d owners", z, owners);
        }
        for (int zt = 0; zt < 20; zt++) if (sw_runs(zt, maxz) != (zt < rows)) printf(" tile row %d is not counted", zt);
        /* a tile row that owns nothing */
        for (int zt = 0; zt < rows; zt++) if (sw_first(zt) > maxz) printf(" tile row %d is empty", zt);
        /* the bottom tile alone holds the box and the unswept row above it */
        if (rows == 1 && maxz + 1 > SW_RZ - 2) printf(" one row does not hold it");
        printf("\n");
    }
    return 0;
}
"""


def test_every_row_has_one_owner(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) == 400
    for line in lines:
        assert len(line.split()) == 2, line
    rows = [int(line.split()[1]) for line in lines]
    assert rows[37] == 1 and rows[38] == 2 and rows[66] == 2 and rows[67] == 3


@pytest.mark.gpu
@pytest.mark.parametrize("top", [34, 35, 36, 37, 38])
def test_box_top_around_the_bottom_tile(gpu, top):
    from baccolonygrowth_b200 import params
    from baccolonygrowth_b200.colony import Colony, packed_colony
    from test_gpu_sweep_block import state
    p = params.parse_parameters(params.shipped_input_text("small"))
    p.box_x, p.box_y, p.box_z, p.box_z_agar, p.max_levels_mg, p.max_cells = 128, 1, 48, 16, 2, 1264
    p.mg_levels = 5
    p = params.finalize(p)
    cells = packed_colony(1200, 60.0, 100.0, seed=7)
    cells["p"][-1], cells["q"][-1] = (-1.0, 0.0, (top - 5 + 0.5) * p.box_length), (1.0, 0.0, (top - 5 + 0.5) * p.box_length)
    a, b = Colony(p, cells), Colony(p, cells)
    for col in (a, b):
        col.initial_density()
        assert col.bbox()[2] == top
    b.set_bbox(*b.bbox())                  # a box of the caller's: single sweeps
    for sweeps, count0 in ((8, 0), (18, 1)):
        la, lb = a.kernel_launches(), b.kernel_launches()
        a.colony_sweeps(sweeps, count0)
        b.colony_sweeps(sweeps, count0)
        assert sweeps == 8 or a.kernel_launches() - la < b.kernel_launches() - lb
        for x, y in zip(state(a), state(b)):
            assert np.array_equal(x, y)
    a.close()
    b.close()
