"""Every thread of a block meets at the same barrier, whichever path its warp takes: fields at rest in part of the grid,
whose warps the strict kernel sends another way than their neighbours'. On the host's build of the tiles (one thread per
CUDA thread; every __syncthreads of the source, and of each of a template's instantiations, is a barrier of its own),
and on the GPU in every output mode, pitched and batched, bit for bit against the oracle."""

import numpy as np
import pytest

import host_tile
from compiler import native
from compiler import workloads as wl
from oracle import api

HOWS = ["none", "all", "w", "south", "column", "top"]


def _fields(geo, nscalar, how):
    arrays = wl.advection_fields(geo, seed=3, nscalar=nscalar).arrays()
    for n, a in enumerate(arrays):
        if how == "all" or (how == "w" and n == 2):
            a[...] = 0.0
        elif how == "south":
            a[:, :a.shape[1] // 2, :] = 0.0
        elif how == "column":
            a[..., a.shape[2] // 2] = -0.0
        elif how == "top":
            a[a.shape[0] // 2:] = 0.0
    return [np.ascontiguousarray(a) for a in arrays]


def _bits(a):
    return np.ascontiguousarray(a).view(np.int64)


def _expected(geo, fields, mode, dt):
    step = api.advection_step(dict(zip("UVW", fields)), geo.dx, geo.dy, geo.dz, geo.halo, fields[3:])
    out = [step[n] for n in ["U", "V", "W", "S0", "S1"][:len(fields)]]
    if mode != native.TENDENCY:
        out = [api.euler(f.copy(), t, dt, geo.halo) for f, t in zip(fields, out)]
    if mode == native.ADVANCE_FILLED:
        out = [api.halo(f, int(n == 2), geo.halo) for n, f in enumerate(out)]
    return out


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("how", HOWS)
def test_on_the_host(how, fast):
    geo = wl.Geometry(33, 11, 5, 1)
    fields = _fields(geo, 1, how)
    same, got = host_tile.step(geo, fields, fast, kz=3)
    assert same, "threads of a block met at different barriers"
    if not fast:
        inner = geo.interior()
        for g, w in zip(got, _expected(geo, fields, native.TENDENCY, 0.0)):
            assert np.array_equal(_bits(g[inner]), _bits(w[inner]))


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("mode", [native.TENDENCY, native.ADVANCE, native.ADVANCE_FILLED])
@pytest.mark.parametrize("how", HOWS)
def test_on_the_gpu(cuda, how, mode, batched):
    geo, pad, dt = wl.Geometry(45, 19, 13, 2), 3, 0.25 * (mode != native.TENDENCY)
    fields = _fields(geo, 2, how)
    wide = lambda a: cuda.nn.functional.pad(cuda.from_numpy(a).cuda(), (0, pad)).contiguous()
    dev = [wide(a) for a in fields]
    out = [cuda.zeros_like(t) for t in dev]
    p, q = [t.data_ptr() for t in dev], [t.data_ptr() for t in out]
    grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz, sx=geo.shape[2] + pad)
    if batched:
        batch = native.Batch([grid], [native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=mode,
                                                         dt=dt)], kz=[4])
        space = cuda.empty(batch.workspace_bytes(), dtype=cuda.uint8, device="cuda")
        batch.prepare(space.data_ptr(), space.numel(), 0)
        batch.step(0)
    else:
        native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=mode, dt=dt)
    cuda.cuda.synchronize()
    inner = geo.interior()
    for g, w in zip(out, _expected(geo, fields, mode, dt)):
        g = g[..., :geo.shape[2]].cpu().numpy()
        if mode != native.ADVANCE_FILLED:
            g, w = g[inner], w[inner]
        assert np.array_equal(_bits(g), _bits(w))
