"""The split step where its vertical solve and its marching divergences change their tiling.

ks_column_ver_tile takes 8 columns and 32 chunks of levels a block up to 1216 columns, 32 columns
and 12 chunks up to 58368 (16 and 16 with FP64 coefficients), and ks_column_ver a thread a column
above; ks_div_h and ks_gas_div cut the column into chunks of at least four levels by the number of
columns.  The grids here lie at those borders and have ragged ends: columns that do not fill the
last block, fewer rows than chunks, one layer more than a whole number of chunks, the fewest and
the most layers.  The bar is tests/test_split.py's against the FP64 step.
"""
import pytest

import cases
import lgame_gpu as L
from test_split import field_errors

# (ny, nx, n_layers, n_oro_layers)
GRIDS = [(3, 5, 3, 2), (19, 65, 13, 12), (32, 38, 33, 25), (65, 97, 128, 96), (243, 240, 5, 4),
         (241, 243, 9, 6)]


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [L.PRECISION_SPLIT, L.PRECISION_SPLIT_FP64_COLUMN])
@pytest.mark.parametrize("grid", GRIDS)
def test_split_close_to_fp64_at_the_tilings_borders(grid, precision):
    ny, nx, nl, no = grid
    n = cases.namelist("jet_1024x1024x80", ny=ny, nx=nx, n_layers=nl, n_oro_layers=no)
    hm = L.HostModel(n)
    states = []
    for prec in (L.PRECISION_FP64, precision):
        cfg = L.config_from_namelist(n)
        cfg.precision = prec
        g = L.GpuModel(cfg, hm.grid)
        for slot in (0, 1):
            g.set_state(slot, hm.state)
        g.set_diag(hm.diag)
        for step in range(2):
            g.pchevi(step % 2, (step + 1) % 2, step)
        states.append(g.get_state(0))
        g.close()
    errs = field_errors(states[1], states[0])
    assert max(errs.values()) <= 1e-5, errs


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [(19, 65, 13, 12), (243, 240, 5, 4)])
def test_split_close_to_fp64_without_a_background_state(grid):
    """Both column kernels without a background state (the thread-per-column one is compiled for each), one
    step, at test_split's bar for it."""
    ny, nx, nl, no = grid
    n = cases.namelist("jet_1024x1024x80", ny=ny, nx=nx, n_layers=nl, n_oro_layers=no, theta_adv_order=2,
                       luse_bg_state=False, lklemp=False)
    hm = L.HostModel(n)
    states = []
    for prec in (L.PRECISION_FP64, L.PRECISION_SPLIT):
        cfg = L.config_from_namelist(n)
        cfg.precision = prec
        g = L.GpuModel(cfg, hm.grid)
        for slot in (0, 1):
            g.set_state(slot, hm.state)
        g.set_diag(hm.diag)
        g.pchevi(0, 1, 0)
        states.append(g.get_state(1))
        g.close()
    errs = field_errors(states[1], states[0])
    assert max(errs.values()) <= 1e-5, errs
