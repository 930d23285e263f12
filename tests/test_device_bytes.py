"""Device memory of a context, on the CPU (the library's host code on a stand-in for the CUDA runtime): the
largest FP64 grid a card takes is what its context leaves.  The bars, in padded fields of the grid, are those of
a step that keeps no metric or work array beside the plain expressions' own: 99.5 dry, 117.5 moist, 152.5 with
the closure and the surface.  And a diagnostic of a closure that is off, which has no device array, is still the
caller's: it comes back as it was set.
"""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
RUN = """
import json, sys
from pathlib import Path
sys.path[:0] = {paths!r}
import numpy as np
import lgame_gpu as L, cases
L.LIB_PATH = Path({lib!r})
n = cases.namelist({config!r}, **json.loads({over!r}))
hm = L.HostModel(n)
cfg = L.config_from_namelist(n)
cfg.precision = L.PRECISION_FP64
g = L.GpuModel(cfg, hm.grid)
field = 8.0 * ((n.ny + 1 + 31) // 32 * 32) * (n.nx + 1) * (n.n_layers + 1)
names = ["tke", "viscosity", "mom_diff_tend_x", "mom_diff_tend_y", "mom_diff_tend_z"]
kept = True
if not cfg.lmom_diff_h:
    assert all(not g.get_diag()[f].any() for f in names)
    d = dict(hm.diag)
    for k, f in enumerate(names):
        d[f] = np.asfortranarray(np.random.default_rng(k).normal(size=d[f].shape))
    g.set_diag(d)
    e = g.get_diag()
    kept = all((d[f] == e[f]).all() for f in names)
print(g.lib.lgame_gpu_device_bytes(g.h) / field, kept)
"""
GRID = dict(ny=94, nx=127, n_layers=20, n_oro_layers=15)
FULL = dict(lmom_diff_h=True, lmom_diff_v=True, ltemp_diff_h=True, ltemp_diff_v=True, lmass_diff_h=True, lmass_diff_v=True,
            lprog_soil_temp=True, nsoillays=5, lsfc_sensible_heat_flux=True, lsfc_phase_trans=True, lpbl=True)
CASES = {"dry": ("rest_hills_512x512x50", {}, 99.5), "moist": ("jet_1024x1024x80", {}, 117.5),
         "physics": ("jet_1024x1024x80", FULL, 152.5)}


@pytest.mark.parametrize("name", CASES)
def test_fp64_context_keeps_to_its_fields(name, recording_library):
    config, over, bar = CASES[name]
    script = RUN.format(paths=[str(HERE), str(HERE.parent / "l-game_gb300")], lib=str(recording_library), config=config,
                        over=json.dumps({**GRID, **over}))
    out = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, env={**os.environ, "OMP_NUM_THREADS": "2"})
    assert out.returncode == 0, out.stderr
    fields, kept = out.stdout.split()
    assert kept == "True"
    assert float(fields) <= bar, fields
