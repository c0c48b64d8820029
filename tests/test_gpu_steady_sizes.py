"""bcg_steady_* on the grid shapes its kernels treat differently, against the
scipy FP64 reference: tiles of 16 and of 32 points a side, grids that end
inside a tile, hierarchies of one level, coarsest levels of few unknowns (one
matrix-vector product) and of many (sweeps in one block, or one launch each
where the level fits no block).  Bounds as in test_steady.py: the field to
1e-10, the gradients to 1e-7 of their largest entry."""
import numpy as np
import pytest

from baccolonygrowth_b200 import steady as st

from steady_ref import SteadyRef

THETA = np.array([0.8, 0.3, 1.0, 0.05])


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,n", [
    (3, 3, 5),          # one level, 6 unknowns
    (9, 3, 20),         # one level, 18 unknowns
    (3, 17, 20),        # one level, tall, 48 unknowns: sweeps
    (17, 9, 0),         # no cells: the field is c0 everywhere
    (33, 17, 400),
    (129, 17, 900),     # coarsest 17 x 3: 34 unknowns, just past the matrix
    (65, 129, 3000),    # taller than wide
    (257, 129, 8000),   # tiles of 32
    (2049, 9, 4000),    # coarsest 513 x 3, in one block
    (2049, 3, 300),     # 2049 x 3: one level in one block
    (4097, 3, 300),     # one level that fits no block: a launch a half-sweep
    (8193, 5, 500),     # the coarsest of two levels fits no block
])
def test_grid_shapes(gpu, nx, nz, n):
    grid = dict(nx=nx, nz=nz, nz_agar=(nz + 1) // 2, h=2.0, c0=20.0)
    cells, w, _ = st.synthetic_problem(nx=nx, nz=nz, nz_agar=grid["nz_agar"], h=2.0, n_cells=n, seed=nx + nz)
    ref = SteadyRef(cells=cells, **grid)
    s = st.Steady(max_cells=max(n, 1), **grid)
    s.set_cells(cells)
    Cr, Cg = ref.solve(THETA, w), s.solve(THETA, w)
    assert np.abs(Cg - Cr).max() <= 1e-10 * np.abs(Cr).max()
    g = np.random.default_rng(nx).standard_normal((nz, nx))
    gtr, gwr = ref.gradients(g)
    gtg, gwg = s.vjp(g)
    if n == 0:
        # a constant field: every difference is 0, and so are the gradients
        # (the reference's direct solve leaves its own rounding in them)
        assert np.array_equal(gtg, np.zeros(4))
    else:
        assert np.abs(gtg - gtr).max() <= 1e-7 * np.abs(gtr).max()
        assert np.abs(gwg - gwr).max() <= 1e-7 * np.abs(gwr).max()
    # a second solve on the same handle (the captured graph) and other parameters
    th = THETA * np.array([1.5, 0.7, 2.0, 3.0])
    assert np.abs(s.solve(th, w) - SteadyRef(cells=cells, **grid).solve(th, w)).max() <= 1e-10 * 20.0
    s.close()
