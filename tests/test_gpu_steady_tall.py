"""bcg_steady_* on a grid with more rows of tiles than a launch has blocks in one
direction (65535): it solves, to a residual worked out here."""
import numpy as np
import pytest

from baccolonygrowth_b200 import steady as st


@pytest.mark.gpu
def test_more_rows_of_tiles_than_blocks(gpu):
    nx, nz, h, c0 = 3, 2 ** 21 + 1, 2.0, 20.0
    d_agar, d_col, vmax, km = 0.8, 0.3, 1e-3, 0.05
    s = st.Steady(nx=nx, nz=nz, nz_agar=2, h=h, c0=c0, max_cells=2)
    k = np.array([3, nz - 2])
    s.set_cells(np.stack([np.full(2, h), k * h, np.full(2, 3.0), np.full(2, 0.5)], 1))
    w = np.array([1.0, 0.7])
    C = s.solve((d_agar, d_col, vmax, km), w, tol=0.5)
    assert s.newton_iters >= 1
    q = np.zeros((nz, nx))
    q[k, 1] = w * 3.0 * 0.5 / (h * h)
    d = np.where(np.arange(nz) < 2, d_agar, d_col)[:, None]

    def residual(C):
        F = -q * vmax * C / (km + C)
        face = np.where(d[1:] == d[:-1], d[1:], 2 * d[1:] * d[:-1] / (d[1:] + d[:-1]))
        dz = face * (C[1:] - C[:-1]) / (h * h)
        F[:-1] += dz
        F[1:] -= dz
        dx = d * (C[:, 1:] - C[:, :-1]) / (h * h)
        F[:, :-1] += dx
        F[:, 1:] -= dx
        F[0] = 0
        return np.abs(F).max()

    assert np.all(C[0] == c0) and np.all(np.isfinite(C))
    assert C[nz - 2, 1] < c0 and C[3, 1] < c0             # both ends were reached
    assert residual(C) <= 0.5 * residual(np.full((nz, nx), c0)) * (1 + 1e-9)
    s.close()
