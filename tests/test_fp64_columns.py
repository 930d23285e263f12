"""The FP64 column solves at the ends of their tiles, against the oracle.

k_column_tracers takes 16 columns and 16 chunks of levels a block: grids whose columns do not
fill the last block, with fewer levels than chunks, with one level more than a whole number of
chunks, and with the most layers a context may have.  The bar is tests/test_gpu_parity.py's
(1e-12 relative per field; the results are the oracle's bits up to c_p_ice's exponential).
"""
import numpy as np
import pytest

import cases
import lgame_gpu as L
import oracle as O

TOL = 1e-12
# (ny, nx, n_layers, n_oro_layers, periodic)
GRIDS = [(3, 5, 3, 2, True), (5, 13, 17, 12, False), (16, 17, 33, 25, True), (65, 97, 128, 96, True)]


@pytest.mark.gpu
@pytest.mark.parametrize("grid", GRIDS)
def test_fp64_columns_match_oracle(grid):
    ny, nx, nl, no, periodic = grid
    kw = dict(n_hills=3, hill_height_min=50.0, hill_height_max=200.0)
    kw.update({} if periodic else dict(lperiodic=False, lfreeslip=False))
    n = cases.namelist("jet_1024x1024x80", ny=ny, nx=nx, n_layers=nl, n_oro_layers=no, **kw)
    hm = L.HostModel(n)
    g = L.GpuModel(L.config_from_namelist(n), hm.grid)
    o = O.Oracle(L.config_from_namelist(n), hm.grid)
    for m in (g, o):
        m.set_state(0, hm.state)
        m.set_state(1, hm.state)
        m.set_diag(hm.diag)
    try:
        for step in range(2):
            for m in (g, o):
                m.pchevi(step % 2, (step + 1) % 2, step)
            a, b = g.get_state((step + 1) % 2), o.get_state((step + 1) % 2)
            da, db = g.get_diag(), o.get_diag()
            bad = [(f, cases.rel_err(a[f], b[f])) for f in L.STATE_FIELDS if not cases.rel_err(a[f], b[f]) <= TOL]
            bad += [(f, cases.rel_err(da[f], db[f])) for f in L.DIAG_FIELDS if not cases.rel_err(da[f], db[f]) <= TOL]
            assert not bad, (step, bad)
            assert all(np.isfinite(v).all() for v in a.values())
    finally:
        g.close()
        o.close()
