"""Fields at rest in part of the grid: the strict kernel's and the stencils' warps that see zeros there take other
paths than their neighbours. Bit for bit against the C oracle."""

import ctypes as c

import numpy as np
import pytest

from compiler import native
from compiler import workloads as wl
from oracle import api

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


def _rest(arrays, how):
    """Zeroes (or flattens) part of the arrays, the first three of which are U, V and W where there are three."""
    for n, a in enumerate(arrays):
        if how == "all" or (how == "w" and n == 2) or (how == "u" and n == 0):
            a[...] = 0.0
        elif how == "south":
            a[..., :a.shape[-2] // 2, :] = 0.0
        elif how == "column":
            a[..., a.shape[-1] // 2] = -0.0
        elif how == "top" and a.ndim == 3:
            a[a.shape[0] // 2:] = 0.0
        elif how == "constant":
            a[...] = 0.25 * (n + 1)
    return arrays


@pytest.mark.parametrize("how", ["all", "w", "u", "south", "column", "top", "constant"])
@pytest.mark.parametrize("shape", [(33, 9, 35), (64, 16, 3)])
def test_strict_step(cuda, how, shape):
    geo = wl.Geometry(*shape, 2)
    fields = wl.advection_fields(geo, seed=3, nscalar=1)
    arrays = _rest(fields.arrays(), how)
    dev = [cuda.from_numpy(a.copy()).cuda() for a in arrays]
    out = [cuda.empty_like(t) for t in dev]
    grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz)
    p, q = [t.data_ptr() for t in dev], [t.data_ptr() for t in out]
    native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:])
    cuda.cuda.synchronize()
    ref = api.advection_step(dict(zip("UVW", arrays)), geo.dx, geo.dy, geo.dz, geo.halo, arrays[3:])
    for name, t in zip(["U", "V", "W", "S0"], out):
        inner = geo.interior()
        assert np.array_equal(_bits(t.cpu().numpy()[inner]), _bits(ref[name][inner])), name


@pytest.mark.parametrize("how", ["all", "south", "column", "top", "constant"])
@pytest.mark.parametrize("dx", [1.0, 0.3])
@pytest.mark.parametrize("n", [(31, 7, 1), (33, 9, 65), (257, 40, 37)])
def test_diffusion(cuda, how, dx, n):
    lib = native.load()
    lib.f2c_diffusion7_v1.argtypes = [c.POINTER(native.Grid), c.c_void_p, c.c_void_p, c.c_double, c.c_double,
                                      c.c_void_p]
    a, = _rest([np.random.default_rng(5).random((n[2] + 2, n[1] + 2, n[0] + 2))], how)
    dev = cuda.from_numpy(a).cuda()
    out = cuda.zeros_like(dev)
    grid = native.make_grid(*n, 1, dx, dx, dx)
    native.check(lib.f2c_diffusion7_v1(c.byref(grid), dev.data_ptr(), out.data_ptr(), 0.1, 1.0, None))
    cuda.cuda.synchronize()
    ref = np.zeros_like(a)
    api.diffusion7(ref, a, 0.1, 1.0, dx, 1)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(ref))


@pytest.mark.parametrize("dx", [0.1, 0.7, 1.0 / 3.0, 1.0 + 2.0**-52, 2.0 - 2.0**-52, 1e-20, 3e45, 1e-90, 1.5 * 2.0**-128])
def test_diffusion_divides(cuda, dx):
    """Quotients by a spacing that is no power of two, within and beyond the range of the two-double reciprocal."""
    lib = native.load()
    lib.f2c_diffusion7_v1.argtypes = [c.POINTER(native.Grid), c.c_void_p, c.c_void_p, c.c_double, c.c_double,
                                      c.c_void_p]
    a = np.random.default_rng(8).random((42, 52, 72)) * 2.0 ** np.random.default_rng(9).integers(-6, 6, (42, 52, 72))
    dev = cuda.from_numpy(a).cuda()
    out = cuda.zeros_like(dev)
    grid = native.make_grid(70, 50, 40, 1, dx, dx, dx)
    native.check(lib.f2c_diffusion7_v1(c.byref(grid), dev.data_ptr(), out.data_ptr(), 0.1 * dx * dx, 1.0, None))
    cuda.cuda.synchronize()
    ref = np.zeros_like(a)
    api.diffusion7(ref, a, 0.1 * dx * dx, 1.0, dx, 1)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(ref))


@pytest.mark.parametrize("how", ["all", "south", "column", "constant"])
@pytest.mark.parametrize("n", [(31, 1), (65, 33), (2000, 700)])
def test_planes(cuda, how, n):
    lib = native.load()
    lib.f2c_jacobi5_v1.argtypes = [c.c_void_p] * 2 + [c.c_int64] * 4 + [c.c_void_p]
    lib.f2c_yee2d_v1.argtypes = [c.c_void_p] * 3 + [c.c_int64] * 4 + [c.c_double] * 2 + [c.c_void_p]
    rng = np.random.default_rng(6)
    fields = _rest([rng.random((n[1] + 2, n[0] + 2)) for _ in range(3)], how)
    dev = [cuda.from_numpy(a.copy()).cuda() for a in fields]
    out = cuda.zeros_like(dev[0])
    native.check(lib.f2c_jacobi5_v1(dev[0].data_ptr(), out.data_ptr(), *n, 1, n[0] + 2, None))
    native.check(lib.f2c_yee2d_v1(*[t.data_ptr() for t in dev], *n, 1, n[0] + 2, 0.5, 0.7, None))
    cuda.cuda.synchronize()
    ref = np.zeros_like(fields[0])
    api.jacobi5(ref, fields[0], 1)
    assert np.array_equal(_bits(out.cpu().numpy()), _bits(ref))
    api.yee2d(*fields, 0.5, 0.7, 1)
    for got, want in zip(dev, fields):
        assert np.array_equal(_bits(got.cpu().numpy()), _bits(want))
