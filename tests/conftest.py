"""pytest configuration: paths to the package and the oracle, and the gpu marker."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
for p in (ROOT / "l-game_gb300", ROOT / "oracle", ROOT / "tests"):
    if str(p) not in sys.path:
        sys.path.insert(0, str(p))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a GB300 (sm_103) GPU and liblgame_gpu.so")


def has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def recording_library(tmp_path_factory):
    """The library's own objects linked with a stand-in for the CUDA runtime (fake_cudart.cpp) that runs no
    kernel: its host code on the CPU."""
    import build
    build.build(force=not list(build.OUT.glob("*.o")))
    objs = sorted(str(p) for p in build.OUT.glob("*.o"))
    assert len(objs) == len(build.CUDA_UNITS) + len(build.CXX_UNITS)
    lib = tmp_path_factory.mktemp("fake") / "liblgame_fake.so"
    cuda = Path(build._nvcc()).resolve().parent.parent
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-fopenmp", f"-I{cuda}/include",
                    str(ROOT / "tests" / "fake_cudart.cpp"), *objs, "-o", str(lib)], check=True)
    return lib
