"""Small kernels of the tests' own (tests/*.cu) around the library's device functions, compiled for the GPU
with a translation unit's flags."""
import ctypes as C
import subprocess
from pathlib import Path

import build

HERE = Path(__file__).resolve().parent


def library(source: str, unit: str, out_dir) -> C.CDLL:
    """tests/<source> compiled with the flags of the library's unit csrc/<unit>."""
    lib = Path(out_dir) / (Path(source).stem + ".so")
    flags = dict(build.CUDA_UNITS)[unit]
    subprocess.run([build._nvcc(), *build.ARCH, *build.NVCC_COMMON, *flags, "-shared", "-cudart", "static",
                    str(HERE / source), "-o", str(lib)], check=True)
    return C.CDLL(str(lib))
