"""The branch-free integer-pipe sum and product of the strict kernels and stencils, and the stencils' points that they
leave to FP64.

``add_rn_range`` and ``mul_rn_range`` (csrc/kernels/soft_fp64.cuh) must equal IEEE addition and multiplication bit for
bit on the operands they take, and leave exactly the others to their caller; the stencils that use them must equal the
oracle bit for bit where neighbouring values are special, far apart or cancel.
"""
import ctypes as c
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from compiler import native
from oracle import api

HERE = Path(__file__).resolve().parent / "soft_fp64"
KERNELS = Path(__file__).resolve().parents[1] / "fortran-to-cuda_gb300" / "csrc" / "kernels"


def test_range_operations_match_ieee(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    fake = tmp_path / "inc"
    fake.mkdir()
    (fake / "cuda_runtime.h").write_text("// empty: the check compiles the header as host C++\n")
    exe = tmp_path / "range_host"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", f"-I{fake}", f"-I{KERNELS}", f"-I{HERE}",
                    str(HERE / "soft_fp64_range_host.cpp"), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe), "1000000"], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout


def _mixed(shape, seed):
    """Random values over 80 binades with runs of equal, opposite, zero, subnormal and huge neighbours."""
    rng = np.random.default_rng(seed)
    a = (rng.random(shape) * 2 - 1) * 2.0 ** rng.integers(-40, 40, shape)
    flat = a.reshape(-1)
    for n, v in enumerate((0.0, -0.0, 1.5, -1.5, 5e-324, -1e-310, 1e300, -1e-300, 2.0 ** 52, 1.0)):
        at = rng.integers(0, flat.size - 4, 12)
        flat[at] = v
        flat[at + 1] = -v if n % 2 else v
    return a


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 1), (33, 9, 2), (64, 8, 33), (65, 17, 31)])
@pytest.mark.parametrize("dx", [1.0, 0.25, 0.3, 2.0 ** -140])
def test_diffusion_of_mixed_values(cuda, shape, dx):
    lib = native.load()
    lib.f2c_diffusion7_v1.argtypes = [c.POINTER(native.Grid), c.c_void_p, c.c_void_p, c.c_double, c.c_double, c.c_void_p]
    nx, ny, nz = shape
    a = _mixed((nz + 2, ny + 2, nx + 2), nx)
    d, out = cuda.from_numpy(a).cuda(), cuda.zeros(a.shape, dtype=cuda.float64, device="cuda")
    grid = native.make_grid(nx, ny, nz, 1, dx, dx, dx)
    dt = 0.125 * dx * dx
    native.check(lib.f2c_diffusion7_v1(c.byref(grid), d.data_ptr(), out.data_ptr(), dt, 1.0, None))
    cuda.cuda.synchronize()
    want = np.zeros(a.shape)
    api.diffusion7(want, a, dt, 1.0, dx, 1)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(want))


@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(1, 1), (63, 31), (64, 33), (130, 9)])
def test_jacobi_and_yee_of_mixed_values(cuda, nx, ny):
    lib = native.load()
    lib.f2c_jacobi5_v1.argtypes = [c.c_void_p] * 2 + [c.c_int64] * 4 + [c.c_void_p]
    lib.f2c_yee2d_v1.argtypes = [c.c_void_p] * 3 + [c.c_int64] * 4 + [c.c_double] * 2 + [c.c_void_p]
    fields = [_mixed((ny + 2, nx + 2), s + nx) for s in range(3)]
    d = [cuda.from_numpy(f).cuda() for f in fields]
    v = cuda.zeros(fields[0].shape, dtype=cuda.float64, device="cuda")
    native.check(lib.f2c_jacobi5_v1(d[0].data_ptr(), v.data_ptr(), nx, ny, 1, nx + 2, None))
    native.check(lib.f2c_yee2d_v1(*[t.data_ptr() for t in d], nx, ny, 1, nx + 2, 0.5, 0.7, None))
    cuda.cuda.synchronize()
    want = np.zeros(fields[0].shape)
    api.jacobi5(want, fields[0], 1)
    assert np.array_equal(_bits(v.cpu().numpy()), _bits(want))
    api.yee2d(*fields, 0.5, 0.7, 1)
    for got, ref in zip(d, fields):
        assert np.array_equal(_bits(got.cpu().numpy()), _bits(ref))
