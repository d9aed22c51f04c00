"""A scalar's infinities and NaN reach its tendency in the fast-fp kernel also where the velocities cancel or are zero
(where its fixed-point sum is zero), as they do in the oracle. On the host's build of the tile, and on the GPU."""

import numpy as np
import pytest

import host_tile
from compiler import native
from compiler import workloads as wl
from oracle import api

FLOWS = {"rest": 0.0, "uniform": 1.0, "negative": -3.0}
GEO = wl.Geometry(34, 10, 5, halo=1)


def _fields(flow, value, everywhere):
    fields = [np.full(GEO.shape, FLOWS[flow]) for _ in range(3)] + [np.full(GEO.shape, 0.5)]
    fields[3][...] = value if everywhere else 0.5
    fields[3][3, 5, 31] = value
    return fields


def _expected(fields, mode, dt):
    with np.errstate(all="ignore"):
        step = api.advection_step(dict(zip("UVW", fields)), GEO.dx, GEO.dy, GEO.dz, GEO.halo, fields[3:])
        want = step["S0"]
        return api.euler(fields[3].copy(), want, dt, GEO.halo) if mode else want


def _same_kind(got, want):
    got, want = got[GEO.interior()], want[GEO.interior()]
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(np.isinf(got), np.isinf(want))
    finite = np.isfinite(want)
    assert (np.abs(got[finite] - want[finite]) <= 1e-12).all()


CASES = [(flow, value, everywhere, mode) for flow in FLOWS for value in (np.nan, np.inf, -np.inf)
         for everywhere in (False, True) for mode in (0, 1)]


@pytest.mark.parametrize("flow,value,everywhere,mode", CASES)
def test_on_the_host(flow, value, everywhere, mode):
    fields = _fields(flow, value, everywhere)
    dt = 0.1 * mode
    _, out = host_tile.step(GEO, fields, True, mode, dt)
    _same_kind(out[3], _expected(fields, mode, dt))


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [False, True])
@pytest.mark.parametrize("flow,value,everywhere,mode", CASES)
def test_on_the_gpu(cuda, flow, value, everywhere, mode, batched):
    fields = _fields(flow, value, everywhere)
    dt = 0.1 * mode
    dev = [cuda.from_numpy(f).cuda() for f in fields]
    out = [cuda.zeros_like(t) for t in dev]
    p, q = [t.data_ptr() for t in dev], [t.data_ptr() for t in out]
    grid = native.make_grid(GEO.nx, GEO.ny, GEO.nz, GEO.halo, GEO.dx, GEO.dy, GEO.dz)
    if batched:
        batch = native.Batch([grid], [native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=mode,
                                                         dt=dt)], tile_rows=4)
        space = cuda.empty(batch.workspace_bytes(), dtype=cuda.uint8, device="cuda")
        batch.prepare(space.data_ptr(), space.numel(), 0)
        batch.set_fast_fp(True)
        batch.step(0)
    else:
        native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=mode, dt=dt, variant=native.FAST)
    cuda.cuda.synchronize()
    _same_kind(out[3].cpu().numpy(), _expected(fields, mode, dt))
