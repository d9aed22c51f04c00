"""Results do not depend on the depth of the z-chunks, bit for bit, whichever outputs are asked for, on fields whose
exponents differ from cell to cell. On the host's build of the tiles, and on the GPU in batches of several depths."""

import numpy as np
import pytest

import host_tile
from compiler import native
from compiler import workloads as wl

GEO = wl.Geometry(35, 10, 7, halo=1)
OUTPUTS = [("UVW", 1), ("UVW", 2), ("U", 0), ("U", 1), ("V", 0), ("V", 1), ("W", 0), ("W", 1), ("", 1)]


def _fields(nscalar):
    rng = np.random.default_rng(21)
    return [(rng.random(GEO.shape) - 0.5) * 2.0 ** rng.integers(-9, 10, GEO.shape) for _ in range(3 + nscalar)]


def _which(names, nscalar):
    return [n in names for n in "UVW"] + [True] * nscalar


def _bits(arrays):
    return [np.ascontiguousarray(a[GEO.interior()]).view(np.int64) for a in arrays]


@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("names,nscalar", OUTPUTS)
def test_on_the_host(names, nscalar, fast):
    fields, which = _fields(nscalar), _which(names, nscalar)
    whole = _bits(host_tile.step(GEO, fields, fast, kz=7, outputs=which)[1])
    for kz in (1, 2, 3):
        chunks = _bits(host_tile.step(GEO, fields, fast, kz=kz, outputs=which)[1])
        assert all(np.array_equal(a, b) for a, b in zip(whole, chunks)), kz


@pytest.mark.gpu
@pytest.mark.parametrize("fast", [True, False])
@pytest.mark.parametrize("names,nscalar", OUTPUTS)
def test_in_batches(cuda, names, nscalar, fast):
    which = _which(names, nscalar)
    dev = [cuda.from_numpy(f).cuda() for f in _fields(nscalar)]
    grid = native.make_grid(GEO.nx, GEO.ny, GEO.nz, GEO.halo, GEO.dx, GEO.dy, GEO.dz)
    p = [t.data_ptr() for t in dev]

    def outputs():
        outs = [cuda.zeros_like(t) if w else None for t, w in zip(dev, which)]
        return outs, [t.data_ptr() if w else None for t, w in zip(outs, which)]

    single, q = outputs()
    native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:],
                     variant=native.FAST if fast else native.FACES)
    for kz in (7, 1, 2, 3):
        for rows in (4, 8, 16) if fast else (8,):
            outs, q = outputs()
            batch = native.Batch([grid], [native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:])],
                                 kz=[kz], tile_rows=rows)
            space = cuda.empty(batch.workspace_bytes(), dtype=cuda.uint8, device="cuda")
            batch.prepare(space.data_ptr(), space.numel(), 0)
            batch.set_fast_fp(fast)
            batch.step(0)
            cuda.cuda.synchronize()
            for a, b in zip(single, outs):
                assert a is None or cuda.equal(a.view(cuda.int64), b.view(cuda.int64)), (kz, rows)
