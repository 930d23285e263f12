"""The order of the split step's kernels across its streams, on the CPU.

The step's host code runs against a stand-in for the CUDA runtime (fake_cudart.cpp, linked to the
library's objects) that records launches, event records and event waits.  From these follows which
launches are ordered; every two launches of which one writes what the other reads or writes have to be.
What each kernel reads and writes is the table below, by substep (a kernel's first and second launch of a
step): prefix "o." the old state, "n." the new one, FP64 and mirror alike.
"""
import json
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
STATE = ("u", "v", "w", "gas", "tr", "th")  # th: rho*theta_v, theta', exner'
FLUX = ["fu", "fv", "gu", "gv"]
ETA = ["ex", "ey", "ez", "uph", "vph", "wph"]
OLD = [f"o.{f}" for f in STATE]
NEW = [f"n.{f}" for f in STATE]
SFC = ["sfc"]


def accesses(name, k, step0):
    """(reads, writes) of launch k (0, 1, ...) of a kernel in a step."""
    rk = "o" if k == 0 else "n"  # the state of the substep
    vec = "o" if step0 and k == 0 else "n"  # of the vector terms: step 0 forms them in both substeps
    X = OLD if rk == "o" else NEW
    table = {
        "k_temperature": (OLD, ["T"]),
        "k_sfc_turb": (OLD + SFC + ["vsq"], SFC),
        "ks_ke": ([f"{vec}.{f}" for f in "uvw"], ["vsq"]),
        "ks_eta": ([f"{vec}.{f}" for f in ("u", "v", "w", "gas")], ETA),
        "ks_vort_flux": ([f"{vec}.w", f"{vec}.gas"] + ETA, ["pvt"]),
        "ks_grad<double>": (["vsq"], ["vsg"]),
        "ks_grad<float>": ([f"{rk}.th"], ["gx", "gy"]),
        "ks_div_h": (["gx", "gy"], ["divf"]),
        "ks_theta_edges": (["o.th", "o.u", "o.v", "divf"], ["tv", "tpe"]),
        "ks_gzp": (["o.th", "o.gas", "o.tr"], ["gzd", "rmz", "gu"]),
        "ks_pgrad": (["o.th", "gzd", "rmz", "gu", "tv", "tpe"], ["pg", "pgcw"]),
        "ks_diff_tke": (OLD + ["tke", "visc", "hdiss"], ["tke_new", "nsq"]),
        "k_diff_zeta": (["o.u", "o.v"], ["zz"]),
        "ks_diff_visc": (OLD + ["T", "tke_new", "zz"], ["vmol", "visc", "vdiv", "tke"]),
        "k_diff_vz": (OLD + ["visc", "zz"], ["vz"]),
        "ks_mom_diff_h": (OLD + ["vz", "vdiv", "mdtz"], ["mdth"]),
        "k_mom_diff_v": (OLD + ["visc", "vmol", "tke", "nsq"], ["mdtz"]),
        "k_pbl": (OLD + SFC + ["vsq"], ["mdth"]),
        "k_diss_rate": (OLD + ["mdth", "mdtz"], ["hdiss"]),
        "k_diff_scalar_col": (OLD + ["T", "visc", "vmol", "tke", "nsq"], ["mdt", "tdh"]),
        "ks_heating_diss": (OLD, ["hdiss"]),
        "k_phase_trans": (OLD + SFC + ["T", "o.soil"], ["ptr", "pth"] + SFC),
        "ks_tend_wind": (["o.u", "o.v", "pg", "pgcw", "vsg", "pvt", "mdth", "mdtz"], ["t.wind", "n.u", "n.v"]),
        "ks_gas_flux": ([f"{rk}.gas", f"{rk}.th", "n.u", "n.v", "tv"], FLUX),
        "ks_theta_flux": (["n.gas", "n.th", "n.u", "n.v", "divf"], FLUX),
        "ks_gas_div": (X + FLUX + ["T", "hdiss", "csh", "mdt", "tdh", "ptr", "pth", "n.u", "n.v"],
                       ["t.gas", "t.rt", "cw"]),
        "ks_tracers": ([f"{rk}.tr", "n.u", "n.v", "cw", "mdt", "ptr"], ["t.tr"]),
        "k_sfc_column_split": (OLD + SFC + [f"{rk}.gas", f"{rk}.th", f"{rk}.w", "o.soil"], ["t.rt", "n.soil"] + SFC),
        "ks_column_ver": (OLD + [f"{rk}.gas", f"{rk}.th", "n.u", "n.v", "t.gas", "t.rt", "t.wind"], ["n.gas", "n.th", "n.w"]),
        "ks_column_ver_tile": (OLD + [f"{rk}.gas", f"{rk}.th", "n.u", "n.v", "t.gas", "t.rt", "t.wind"],
                               ["n.gas", "n.th", "n.w"]),
        "ks_column_tracers": (["o.tr", "o.gas", "o.w", "n.w", "t.tr", "T"], ["n.tr", "csh_part"]),
        "ks_csh_sum": (["csh_part"], ["csh"]),
    }
    return table[name]


def unordered(log):
    """The pairs of launches that touch the same array, one of them writing it, with no order between
    them.  Two steps, the second from what is the first's new state."""
    clocks, events, launches, count = {}, {}, [], {}
    for line in log:
        what, stream, rest = line.split(" ", 2)
        own = clocks.setdefault(stream, set())
        if what == "record":
            events[rest] = set(own)
        elif what == "wait":
            own |= events.get(rest, set())
        elif what == "launch":
            if rest == "k_temperature":  # a step begins
                step = count.get("step", -1) + 1
                count = {"step": step}
            k = count.get(rest, 0)
            count[rest] = k + 1
            reads, writes = accesses(rest, k, count["step"] == 0)
            slot = {"o": f"s{count['step'] % 2}", "n": f"s{(count['step'] + 1) % 2}"}
            place = lambda names: {re.sub(r"^([on])\.", lambda m: slot[m[1]] + ".", n) for n in names}
            launches.append((f"step {count['step']} {rest} #{k}", place(reads), place(writes), set(own)))
            own.add(len(launches) - 1)
    bad = []
    for b, (nb, rb, wb, before) in enumerate(launches):
        for a in range(b):
            na, ra, wa, _ = launches[a]
            shared = (wa & (rb | wb)) | (ra & wb)
            if shared and a not in before:
                bad.append((na, nb, sorted(shared)))
    return bad, len(launches)


RUN = """
import ctypes as C, json, sys
from pathlib import Path
sys.path[:0] = {paths!r}
import lgame_gpu as L, cases
L.LIB_PATH = Path({lib!r})
key, over = cases.SMALL[{small!r}]
n = cases.namelist(key, **dict(over, **json.loads({over!r})))
hm = L.HostModel(n)
cfg = L.config_from_namelist(n)
cfg.precision, cfg.check_finite = L.PRECISION_SPLIT, 0
g = L.GpuModel(cfg, hm.grid)
g.set_graphs(False)
lib = L.load_library()
lib.fake_log.restype = C.c_char_p
g.pchevi(0, 1, 0)  # (with the mirrors' refresh)
lib.fake_clear()
for step in range(2):
    g.pchevi(step % 2, (step + 1) % 2, step)
print(lib.fake_log().decode())
"""


PHYSICS = dict(lmom_diff_h=True, lmom_diff_v=True, ltemp_diff_h=True, ltemp_diff_v=True, lmass_diff_h=True,
               lmass_diff_v=True, lprog_soil_temp=True, lsfc_sensible_heat_flux=True, lsfc_phase_trans=True, lpbl=True,
               lphase_trans=True)
CASES = {
    "plain": ("jet", {}),
    "linear": ("jet", dict(llinear=True, lcorio=False)),
    "second_order": ("jet", dict(theta_adv_order=2)),
    "physics": ("jet", PHYSICS),
    "dry": ("schaer", {}),
}


@pytest.mark.parametrize("name", CASES)
def test_launches_that_share_an_array_are_ordered(name, recording_library):
    small, over = CASES[name]
    script = RUN.format(paths=[str(HERE), str(HERE.parent / "l-game_gb300")], lib=str(recording_library),
                        small=small, over=json.dumps(over))
    out = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, env={**os.environ, "OMP_NUM_THREADS": "2"})
    assert out.returncode == 0, out.stderr
    log = []
    for line in out.stdout.splitlines():
        if line.startswith("launch"):
            what, stream, mangled = line.split(" ", 2)
            # the kernel's own name, and the scalar's type where the table tells them apart
            m = re.search(r"\d+(ks?_[a-z_]+[a-z])(I[fd]Lb)?", mangled)
            kernel = m[1] + ({"IfLb": "<float>", "IdLb": "<double>"}[m[2]] if m[1] == "ks_grad" else "")
            line = f"{what} {stream} {kernel}"
        if line:
            log.append(line)
    bad, launches = unordered(log)
    assert launches >= 2 * 17 and len({line.split()[1] for line in log}) >= 2
    assert not bad, bad
