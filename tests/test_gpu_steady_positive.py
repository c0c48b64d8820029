"""bcg_steady_* on a field that stays positive (the uptake's linearisation counts,
where a strong uptake drives the field far below zero and leaves the Laplacian),
against the scipy FP64 reference, at the bounds of test_gpu_steady_sizes.py."""
import numpy as np
import pytest

from baccolonygrowth_b200 import steady as st

from steady_ref import SteadyRef

THETA = np.array([0.8, 0.3, 3e-4, 0.05])


@pytest.mark.gpu
@pytest.mark.parametrize("nx,nz,n", [(17, 9, 100), (65, 33, 4000), (129, 65, 50000), (257, 129, 20000)])
def test_positive_field(gpu, nx, nz, n):
    grid = dict(nx=nx, nz=nz, nz_agar=(nz + 1) // 2, h=2.0, c0=20.0)
    cells, w, _ = st.synthetic_problem(nx=nx, nz=nz, nz_agar=grid["nz_agar"], h=2.0, n_cells=n, seed=nx)
    ref, s = SteadyRef(cells=cells, **grid), st.Steady(max_cells=n, **grid)
    s.set_cells(cells)
    Cr, Cg = ref.solve(THETA, w), s.solve(THETA, w)
    assert 0 < Cr.min() < 20.0
    assert np.abs(Cg - Cr).max() <= 1e-10 * np.abs(Cr).max()
    g = np.random.default_rng(nx).standard_normal((nz, nx))
    (gtr, gwr), (gtg, gwg) = ref.gradients(g), s.vjp(g)
    assert np.abs(gtg - gtr).max() <= 1e-7 * np.abs(gtr).max()
    assert np.abs(gwg - gwr).max() <= 1e-7 * np.abs(gwr).max()
    s.close()
