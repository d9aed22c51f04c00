"""The fast-fp kernel where one velocity component is far larger than the others: its tendency is then a small
difference of large values. On the host's build of the tile, and on the GPU.

The bound: five roundings of the result or its coefficient, 2^-50 of it, and 27 units of 2^-56 times the power of two
above the largest component value P and that above the largest D of the velocities across and of the difference along
(wide_int.cuh); each power is at most twice the value, so 27 * 4 * 2^-56 < 2^-49 of their product.
"""
import numpy as np
import pytest

import host_tile
from compiler import native
from compiler import workloads as wl
from oracle import api
from tolerance import check

X = np.longdouble  # 64 bits of significand or more; the expressions below cancel no large products
SPACINGS = [(10.0, 10.0, 5.0), (10.0, 7.0, 3.0)]
CROSS = [1e-1, 1e-3, 1e-6, 1e-9, 1e-13, 0.0]


def _flow(component, cross, own, spacing):
    """One component 10 (with noise `own`), the others noise of size `cross`, and a scalar."""
    geo = wl.Geometry(34, 10, 5, 1, *spacing)
    rng = np.random.default_rng(11)
    fields = [(rng.random(geo.shape) * 2 - 1) * cross for _ in range(3)] + [rng.random(geo.shape)]
    fields[component] = 10.0 + (rng.random(geo.shape) * 2 - 1) * own
    return geo, fields


def _expected(geo, fields, n):
    """The tendency of component n, and the bound's product P D times its coefficient."""
    h, d = geo.halo, (geo.dx, geo.dy, geo.dz)

    def at(f, *moves):
        o = [h, h, h]
        for axis, by in moves:
            o[axis] += by
        return fields[f][o[2]:o[2] + geo.nz, o[1]:o[1] + geo.ny, o[0]:o[0] + geo.nx].astype(X)

    c, want, largest = at(n), X(0), 0.0
    for axis in range(3):
        f1, f0 = at(n, (axis, 1)), at(n, (axis, -1))
        if axis == n:
            want = want - X(0.125) / X(d[axis]) * (f1 - f0) * (f1 + f0 + 4 * c)
            largest = max(largest, float(np.abs(f1 - f0).max()) / d[axis])
        else:
            q, qn = at(axis) + at(axis, (n, 1)), at(axis, (axis, -1)) + at(axis, (axis, -1), (n, 1))
            want = want - X(0.0625) / X(d[axis]) * (2 * (f1 - f0) * (q + qn) + (f1 + f0 + 2 * c) * (q - qn))
            largest = max(largest, float(np.abs(fields[axis]).max()) / d[axis])
    return want, 0.0625 * float(np.abs(fields[n]).max()) * largest


def _verify(geo, fields, component, own, got):
    got = [np.ascontiguousarray(g[geo.interior()]) for g in got]
    for n in range(3):
        want, unit = _expected(geo, fields, n)
        assert (np.abs(got[n].astype(X) - want) <= 2.0 ** -50 * np.abs(want) + 2.0 ** -49 * unit).all(), n
    if own == 0.0:  # (with noise along itself the oracle's own fluxes cancel)
        ref = api.advection_step(dict(zip("UVW", fields)), geo.dx, geo.dy, geo.dz, geo.halo, fields[3:])
        for name, g in zip(["U", "V", "W", "S0"], got):
            check(g, ref[name][geo.interior()], name)


@pytest.mark.parametrize("spacing", SPACINGS)
@pytest.mark.parametrize("cross", CROSS)
@pytest.mark.parametrize("component", [0, 1, 2])
def test_on_the_host(component, cross, spacing):
    for own in (0.0, cross):
        geo, fields = _flow(component, cross, own, spacing)
        _verify(geo, fields, component, own, host_tile.step(geo, fields, True)[1])


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [0, 4])
@pytest.mark.parametrize("spacing", SPACINGS)
@pytest.mark.parametrize("cross", CROSS)
@pytest.mark.parametrize("component", [0, 1, 2])
def test_on_the_gpu(cuda, component, cross, spacing, rows):
    for own in (0.0, cross):
        geo, fields = _flow(component, cross, own, spacing)
        dev = [cuda.from_numpy(f).cuda() for f in fields]
        out = [cuda.zeros_like(t) for t in dev]
        p, q = [t.data_ptr() for t in dev], [t.data_ptr() for t in out]
        grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz)
        if rows:
            batch = native.Batch([grid], [native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:])],
                                 tile_rows=rows)
            space = cuda.empty(batch.workspace_bytes(), dtype=cuda.uint8, device="cuda")
            batch.prepare(space.data_ptr(), space.numel(), 0)
            batch.step(0)
        else:
            native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], variant=native.FAST)
        cuda.cuda.synchronize()
        _verify(geo, fields, component, own, [t.cpu().numpy() for t in out])
