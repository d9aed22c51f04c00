"""The advection tiles of the CUDA headers on the host (host_tile.cpp): compiled with the host's C++ compiler, called
with numpy arrays of shape (nz+2h, ny+2h, nx+2h)."""

import ctypes
import shutil
import subprocess
from functools import lru_cache
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
KERNELS = HERE.parents[1] / "fortran-to-cuda_gb300" / "csrc" / "kernels"
BUILD = HERE / "_build"


@lru_cache(maxsize=1)
def library():
    """The compiled tiles; the calling test is skipped where there is no host compiler."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    BUILD.mkdir(exist_ok=True)
    target = BUILD / "libhost_tile.so"
    subprocess.run([cxx, "-O2", "-std=c++20", "-ffp-contract=off", "-w", "-fPIC", "-shared", "-pthread",
                    f"-I{HERE}", f"-I{KERNELS}", str(HERE / "host_tile.cpp"), "-o", str(target)], check=True)
    return ctypes.CDLL(str(target))


def _pointers(arrays):
    return (ctypes.c_void_p * len(arrays))(*[None if a is None else a.ctypes.data for a in arrays])


def _call(function, geo, fields, outputs, *rest):
    outs = [np.full_like(f, np.nan) if w else None for f, w in zip(fields, outputs)]
    size = (ctypes.c_int * 4)(geo.nx, geo.ny, geo.nz, geo.halo)
    spacing = (ctypes.c_double * 3)(geo.dx, geo.dy, geo.dz)
    status = function(_pointers(fields), _pointers(outs), len(fields) - 3, size, spacing, *rest)
    return status, [o for o in outs if o is not None]


def step(geo, fields, fast, mode=0, dt=0.0, kz=32, outputs=None):
    """One step of the fast-fp or the strict tile: whether every block met at one barrier at a time, and the padded
    outputs (NaN where nothing was written)."""
    run = lambda *a: library().host_step(int(fast), *a)
    status, outs = _call(run, geo, fields, outputs or [True] * len(fields), mode, ctypes.c_double(dt), kz)
    assert status != 2, "no such instantiation"
    return status == 0, outs


def fp64_form(geo, fields, mode=0, dt=0.0):
    """The fast-fp kernel's FP64 form at every point."""
    return _call(library().host_fp64_form, geo, fields, [True] * len(fields), mode, ctypes.c_double(dt))[1]
