"""bcg_steady_solve's report of its Newton steps: fewer than 50 where the bound
was met, 50 where it was not (here one below F's rounding), with the field of
the last step."""
import numpy as np
import pytest

from baccolonygrowth_b200 import steady as st

from steady_ref import SteadyRef

THETA = np.array([0.8, 0.3, 1.0, 0.05])


@pytest.mark.gpu
def test_newton_steps_reported(gpu):
    grid = dict(nx=17, nz=9, nz_agar=5, h=2.0, c0=20.0)
    cells, w, _ = st.synthetic_problem(nx=17, nz=9, nz_agar=5, h=2.0, n_cells=200, seed=4)
    ref = SteadyRef(cells=cells, **grid).solve(THETA, w)
    s = st.Steady(max_cells=200, **grid)
    s.set_cells(cells)
    for tol, bound in ((1e-10, 1e-6), (1e-300, 1e-10)):
        C = s.solve(THETA, w, tol=tol)
        assert (s.newton_iters < 50) == (tol > 1e-300)
        assert np.abs(C - ref).max() <= bound * np.abs(ref).max()
    s.close()
