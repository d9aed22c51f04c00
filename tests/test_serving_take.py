"""Results taken from the server (f2c_serve_take_v1): handed over once, alive after the server, refused afterwards."""
import ctypes

import numpy as np
import pytest

from compiler import native, serving
from compiler.resident.domain import ResidentDomain

STALE = 2  # FORT_SCOPE_STALE


@pytest.mark.gpu
@pytest.mark.parametrize("shape,nscalar", [((1, 1, 3), 0), ((33, 20, 9), 2)])
def test_a_field_is_taken_once_and_outlives_the_server(cuda, shape, nscalar):
    lib = native.runtime()
    dom = ResidentDomain(lib, fast_fp=True)
    dom.begin_epoch(device=0)
    dom.require(lib.fort_scope_host_pinning_set_v1(dom.context, 0))
    opts = native.ServeOptions(version=native.SERVE_ABI_VERSION, max_active=4, depth=2, tick_points=1 << 62)
    handle, ident, count = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_size_t()
    dom.require(lib.f2c_serve_create_v1(dom.context, ctypes.byref(opts), ctypes.byref(handle)))
    nx, ny, nz = shape
    spec = native.ServeJob(nx=nx, ny=ny, nz=nz, halo=1, dx=10.0, dy=10.0, dz=5.0, dt=0.01, nscalar=nscalar, steps=2,
                           seed=3, arrival=0.0, flags=native.SERVE_KEEP_RESULT)
    dom.require(lib.f2c_serve_submit_v1(handle.value, ctypes.byref(spec), ctypes.byref(ident)))
    dom.require(lib.f2c_serve_drain_v1(handle.value, -1.0))
    take = lambda f, p: lib.f2c_serve_take_v1(handle.value, ident.value, f, ctypes.byref(p))
    lent, mine = ctypes.POINTER(ctypes.c_double)(), ctypes.c_void_p()
    assert take(3 + nscalar, mine) != 0 and take(-1, mine) != 0 and not mine.value
    assert lib.f2c_serve_take_v1(handle.value, ident.value + 1, 0, ctypes.byref(mine)) == STALE
    padded = (nz + 2, ny + 2, nx + 2)
    copies, taken = [], []
    for f in range(3 + nscalar):
        dom.require(lib.f2c_serve_result_v1(handle.value, ident.value, f, ctypes.byref(lent)))
        copies.append(np.ctypeslib.as_array(lent, shape=padded).copy())
        assert take(f, mine) == 0
        taken.append(np.asarray(serving._Taken(lib, mine.value, padded)))
        assert take(f, mine) == STALE
        assert lib.f2c_serve_result_v1(handle.value, ident.value, f, ctypes.byref(lent)) == STALE
    dom.require(lib.f2c_serve_release_v1(handle.value, ident.value))
    assert take(0, mine) == STALE
    dom.require(lib.f2c_serve_destroy_v1(handle.value))
    dom.close()
    for a, b in zip(taken, copies):
        view = a[1:-1]  # keeps the memory
        assert a.flags.writeable and np.array_equal(a.view(np.int64), b.view(np.int64))
        del a
        view[...] = 1.0
