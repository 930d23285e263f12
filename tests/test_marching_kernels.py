"""The split step's kernels that march down chunks of levels (ks_eta, ks_vort_flux, ks_grad, ks_diff_tke,
ks_diff_visc, ks_mom_diff_h), field by field against the FP64 step, whose kernels have none of their tiling.

The grids have ragged ends in every direction: rows one short of, at and one past a warp (the
extra row ny+1 starts a new one), columns likewise of a block's four, layers that leave a last chunk
of one to three; periodic, and between boundaries whose edges no operator writes.  A point that takes a wrong
neighbour, level or branch is off by the size of the field.  The bar: FP32 terms are rounded to 6e-8,
at most some thirty are added, and the differences taken (of winds, heights and viscosities over a
cell or layer) lose at most a factor of a thousand: 30*6e-8*1000 = 2e-3 of the field's maximum.
"""
import numpy as np
import pytest

import cases
import lgame_gpu as L

FIELDS = ["pot_vort_tend_x", "pot_vort_tend_y", "pot_vort_tend_z", "v_squared_grad_x", "v_squared_grad_y",
          "v_squared_grad_z", "tend_wind_u", "tend_wind_v", "tke", "viscosity", "mom_diff_tend_x", "mom_diff_tend_y"]
DIFF = dict(lmom_diff_h=True, lmom_diff_v=True, ltemp_diff_h=True, ltemp_diff_v=True, lmass_diff_h=True,
            lmass_diff_v=True)
# (ny, nx, n_layers, n_oro_layers)
GRIDS = [(31, 5, 9, 7), (32, 7, 13, 12), (33, 6, 24, 18), (19, 36, 33, 25)]


@pytest.mark.gpu
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("grid", GRIDS)
def test_marching_kernels_close_to_fp64(grid, periodic):
    ny, nx, nl, no = grid
    n = cases.namelist("jet_1024x1024x80", ny=ny, nx=nx, n_layers=nl, n_oro_layers=no, dx=5000.0, dy=5000.0, n_hills=5,
                       hill_width_min=8000.0, hill_width_max=20000.0, lperiodic=periodic, lfreeslip=periodic, **DIFF)
    hm = L.HostModel(n)
    rng = np.random.default_rng(1)
    state = dict(hm.state)
    for f in ("wind_u", "wind_v"):  # smooth along each axis, so that every difference has its part
        s = hm.state[f].shape
        a, b, c = (np.sin(2 * np.pi * (np.arange(m) / max(m - (m in (ny + 1, nx + 1)), 1) + rng.random())) for m in s)
        state[f] = np.asfortranarray(hm.state[f] + 3.0 * a[:, None, None] * b[None, :, None] + 2.0 * c[None, None, :])
    diags = []
    for prec in (L.PRECISION_FP64, L.PRECISION_SPLIT):
        cfg = L.config_from_namelist(n)
        cfg.precision = prec
        g = L.GpuModel(cfg, hm.grid)
        for slot in (0, 1):
            g.set_state(slot, state)
        g.set_diag(hm.diag)
        for step in range(2):
            g.pchevi(step % 2, (step + 1) % 2, step)
        diags.append(g.get_diag())
        g.close()
    for f in FIELDS:
        a, b = diags[1][f], diags[0][f]
        assert np.isfinite(b).all() and np.abs(b).max() > 0.0, f
        assert np.abs(a - b).max() <= 2e-3 * np.abs(b).max(), (f, float(np.abs(a - b).max() / np.abs(b).max()))
