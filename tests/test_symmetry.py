"""A flow that does not vary along y keeps that symmetry in the split step: every row stays the first one's copy
and the wind along y exactly zero, as in the FP64 step.  The terms of a circulation cancel there only if each of
their products is rounded by itself; one left inside a multiply-add drives a wind along y of its own (2.7e-6 m/s
after 6 h of the Schaer wave), which the closure amplifies."""
import numpy as np
import pytest

import cases
import lgame_gpu as L

DIFF = dict(lmom_diff_h=True, lmom_diff_v=True, ltemp_diff_h=True, ltemp_diff_v=True, lmass_diff_h=True,
            lmass_diff_v=True)


@pytest.mark.gpu
@pytest.mark.parametrize("over", [{}, DIFF], ids=["plain", "closure"])
@pytest.mark.parametrize("precision", [L.PRECISION_FP64, L.PRECISION_SPLIT])
def test_rows_of_a_slice_stay_the_same(precision, over):
    key, small = cases.SMALL["schaer"]
    n = cases.namelist(key, **{**small, **over})
    hm = L.HostModel(n)
    cfg = L.config_from_namelist(n)
    cfg.precision = precision
    g = L.GpuModel(cfg, hm.grid)
    for slot in (0, 1):
        g.set_state(slot, hm.state)
    g.set_diag(hm.diag)
    for step in range(50):
        g.pchevi(step % 2, (step + 1) % 2, step)
    s = g.get_state(0)
    g.close()
    assert np.abs(s["wind_w"]).max() > 1e-3 and not s["wind_v"].any()
    for f in L.ATMOS_FIELDS:
        np.testing.assert_array_equal(s[f], np.broadcast_to(s[f][:1], s[f].shape), err_msg=f)
