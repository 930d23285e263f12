"""The linear model (llinear: no vorticity in the wind tendency, no kinetic energy gradient), with and without the
Coriolis force, which then is all that the vorticity flux carries: the FP64 step against the oracle at
tests/test_gpu_parity.py's bar, the split step against the FP64 step at tests/test_split.py's, and its
concurrent branches against the serial order, bit for bit."""
import numpy as np
import pytest

import cases
import lgame_gpu as L
import oracle as O
from test_split import field_errors

BOUNDS = [dict(), dict(lperiodic=False, lfreeslip=False)]


def model(n, hm, precision, graphs=True, serial=False):
    cfg = L.config_from_namelist(n)
    cfg.precision = precision
    g = L.GpuModel(cfg, hm.grid)
    g.set_graphs(graphs)
    g.set_profiling(serial)
    for slot in (0, 1):
        g.set_state(slot, hm.state)
    g.set_diag(hm.diag)
    return g


def linear_case(coriolis, bounds):
    key, over = cases.SMALL["jet"]
    n = cases.namelist(key, **{**over, **bounds, "llinear": True, "lcorio": coriolis})
    return n, L.HostModel(n)


@pytest.mark.gpu
@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("coriolis", [False, True])
def test_linear_fp64_step_matches_oracle(coriolis, bounds):
    n, hm = linear_case(coriolis, bounds)
    g, o = model(n, hm, L.PRECISION_FP64), O.Oracle(L.config_from_namelist(n), hm.grid)
    for slot in (0, 1):
        o.set_state(slot, hm.state)
    o.set_diag(hm.diag)
    for step in range(2):
        for m in (g, o):
            m.pchevi(step % 2, (step + 1) % 2, step)
        a, b = g.get_state((step + 1) % 2), o.get_state((step + 1) % 2)
        da, db = g.get_diag(), o.get_diag()
        bad = [(f, cases.rel_err(a[f], b[f])) for f in L.STATE_FIELDS if not cases.rel_err(a[f], b[f]) <= 1e-12]
        bad += [(f, cases.rel_err(da[f], db[f])) for f in L.DIAG_FIELDS if not cases.rel_err(da[f], db[f]) <= 1e-12]
        assert not bad, (step, bad)
    assert np.abs(db["v_squared_grad_x"]).max() == 0.0
    assert (np.abs(db["pot_vort_tend_x"]).max() > 0.0) == coriolis
    g.close()
    o.close()


@pytest.mark.gpu
@pytest.mark.parametrize("bounds", BOUNDS)
@pytest.mark.parametrize("coriolis", [False, True])
def test_linear_split_step_close_to_fp64(coriolis, bounds):
    n, hm = linear_case(coriolis, bounds)
    states = []
    for precision in (L.PRECISION_FP64, L.PRECISION_SPLIT):
        g = model(n, hm, precision)
        for step in range(2):
            g.pchevi(step % 2, (step + 1) % 2, step)
        states.append(g.get_state(0))
        g.close()
    errs = field_errors(states[1], states[0])
    assert max(errs.values()) <= 1e-5, errs


@pytest.mark.gpu
def test_linear_split_branches_equal_serial_order():
    n, hm = linear_case(False, {})
    models = [model(n, hm, L.PRECISION_SPLIT, graphs=False, serial=serial) for serial in (False, True)]
    for step in range(5):
        for g in models:
            g.pchevi(step % 2, (step + 1) % 2, step)
    a, b = (g.get_state(1) for g in models)
    for f in L.STATE_FIELDS:
        assert np.isfinite(a[f]).all(), f
        np.testing.assert_array_equal(a[f], b[f], err_msg=f)
    for g in models:
        g.close()
