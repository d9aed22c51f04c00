"""Diffusion of plateaus, whose points keep their value without the last product: values and factors at the ends of what
the shortcut takes, bit for bit against the C oracle (a NaN is a NaN)."""
import ctypes as c

import numpy as np
import pytest

from compiler import native
from oracle import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [0.75, -3.0, 2.0**-511, 2.0**-512, 2.0**511, -(2.0**512), 5e-324, np.inf])
@pytest.mark.parametrize("dx", [1.0, 0.3, 2.0**-128, 2.0**-129, 1e-200])
@pytest.mark.parametrize("nu", [1.0, -0.5, 0.0, 1e-300, np.inf, np.nan])
def test_plateaus(cuda, value, dx, nu):
    lib = native.load()
    lib.f2c_diffusion7_v1.argtypes = [c.POINTER(native.Grid), c.c_void_p, c.c_void_p, c.c_double, c.c_double, c.c_void_p]
    nx, ny, nz = 41, 11, 5
    a = np.full((nz + 2, ny + 2, nx + 2), value)
    a[:, :, 20:30] = 1.5 * value  # a second plateau, and between them points that are done in full
    a[3, 5, 7] = -value
    dev = cuda.from_numpy(a).cuda()
    out = cuda.zeros_like(dev)
    grid = native.make_grid(nx, ny, nz, 1, dx, dx, dx)
    native.check(lib.f2c_diffusion7_v1(c.byref(grid), dev.data_ptr(), out.data_ptr(), 0.125, nu, None))
    cuda.cuda.synchronize()
    want = np.zeros_like(a)
    with np.errstate(all="ignore"):
        api.diffusion7(want, a, 0.125, nu, dx, 1)
    got = out.cpu().numpy()
    assert ((got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))).all()
