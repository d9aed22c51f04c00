"""The fast-fp kernel's 64-bit fixed-point arithmetic: its error bound against extended precision, the ends of its
tiles, and the values it leaves to FP64.

The bound (csrc/kernels/wide_int.cuh): five roundings of the result or its coefficient, 2^-50 of it, and 27 units of 2^-56 times the
powers of two above the largest component value and the largest scaled velocity of the stencil; each power is at most
twice the value, so 27 * 4 * 2^-56 < 2^-49 of their product (the maxima over the whole field here).
"""
import numpy as np
import pytest

from compiler import native
from compiler import workloads as wl
from oracle import api

pytestmark = pytest.mark.gpu
X = np.longdouble  # 64 bits of significand or more on both machines


def _launch(torch, fields, geo, mode=native.TENDENCY, dt=0.0):
    ins = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in fields]
    outs = [torch.full_like(t, float("nan")) for t in ins]
    grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz)
    p, q = [t.data_ptr() for t in ins], [t.data_ptr() for t in outs]
    native.advection(grid, *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=mode, dt=dt, variant=native.FAST)
    torch.cuda.synchronize()
    return [o.cpu().numpy()[geo.interior()] for o in outs]


def _extended(fields, geo):
    """The tendencies in extended precision, the component's expression of the source with the axes exchanged."""
    h = geo.halo

    def at(f):
        f = f.astype(X)
        return lambda i, j, k: f[h + k:h + k + geo.nz, h + j:h + j + geo.ny, h + i:h + i + geo.nx]

    def turned(f, order):
        return lambda *o: f(*(o[n] for n in order))

    def component(u, v, w, d):
        a = [X(0.25) / X(x) for x in d]
        c = u(0, 0, 0)
        div = a[0] * ((u(1, 0, 0) + c) ** 2 - (c + u(-1, 0, 0)) ** 2) \
            + a[1] * ((u(0, 1, 0) + c) * (v(1, 0, 0) + v(0, 0, 0)) - (c + u(0, -1, 0)) * (v(1, -1, 0) + v(0, -1, 0))) \
            + a[2] * ((u(0, 0, 1) + c) * (w(1, 0, 0) + w(0, 0, 0)) - (c + u(0, 0, -1)) * (w(1, 0, -1) + w(0, 0, -1)))
        adv = 2 * a[0] * (u(1, 0, 0) - u(-1, 0, 0)) * c \
            + a[1] / 2 * (u(0, 1, 0) - u(0, -1, 0)) * (v(0, 0, 0) + v(1, 0, 0) + v(0, -1, 0) + v(1, -1, 0)) \
            + a[2] / 2 * (u(0, 0, 1) - u(0, 0, -1)) * (w(0, 0, 0) + w(1, 0, 0) + w(0, 0, -1) + w(1, 0, -1))
        return -(div + adv) / 2

    u, v, w = (at(f) for f in fields[:3])
    dx, dy, dz = geo.dx, geo.dy, geo.dz
    out = [component(u, v, w, (dx, dy, dz)),
           component(*(turned(f, (1, 0, 2)) for f in (v, u, w)), (dy, dx, dz)),
           component(*(turned(f, (2, 1, 0)) for f in (w, v, u)), (dz, dy, dx))]
    for s in map(at, fields[3:]):
        c = s(0, 0, 0)
        out.append(-X(0.5) * ((u(0, 0, 0) * (s(1, 0, 0) + c) - u(-1, 0, 0) * (c + s(-1, 0, 0))) / X(dx)
                              + (v(0, 0, 0) * (s(0, 1, 0) + c) - v(0, -1, 0) * (c + s(0, -1, 0))) / X(dy)
                              + (w(0, 0, 0) * (s(0, 0, 1) + c) - w(0, 0, -1) * (c + s(0, 0, -1))) / X(dz)))
    return out


def _velocity(fields, geo):
    """The largest |velocity| / spacing, times the coefficient 0.0625 (a component's) of the direction."""
    return max(float(np.abs(f).max()) / d for f, d in zip(fields[:3], (geo.dx, geo.dy, geo.dz)))


@pytest.mark.parametrize("shape,halo,nscalar", [((1, 1, 1), 1, 0), ((32, 8, 1), 1, 1), ((31, 7, 3), 2, 4),
                                                ((33, 9, 2), 1, 2), ((65, 17, 34), 2, 3), ((64, 16, 33), 1, 0)])
@pytest.mark.parametrize("spacing", [(10.0, 10.0, 5.0), (10.0, 7.0, 3.0)])
def test_error_bound_at_tile_ends(cuda, shape, halo, nscalar, spacing):
    geo = wl.Geometry(*shape, halo, *spacing)
    rng = np.random.default_rng(sum(shape) + nscalar)
    fields = [(rng.random(geo.shape) * 2 - 1) * scale for scale in (8.0, 1.0, 1e-3, 300.0, 1.0, 1e-20, 5.0)[:3 + nscalar]]
    q = _velocity(fields, geo)
    for n, (got, want) in enumerate(zip(_launch(cuda, fields, geo), _extended(fields, geo))):
        # a scalar's coefficient 0.5/d is eight times a component's
        unit = 0.0625 * (8 if n > 2 else 1) * float(np.abs(fields[n]).max()) * q
        bound = 2.0 ** -50 * np.abs(want) + 2.0 ** -49 * unit
        assert np.isfinite(got).all()
        assert (np.abs(got.astype(X) - want) <= bound).all(), n


@pytest.mark.parametrize("mode,dt", [(native.TENDENCY, 0.0), (native.ADVANCE, 0.1)])
def test_values_left_to_fp64(cuda, mode, dt):
    """Infinities, NaN, subnormals, zeros and both ends of the exponent range among ordinary values: finite exactly
    where the oracle is, and there within the tolerance of the contract (1e-12 of the stencil's largest product)."""
    geo = wl.Geometry(40, 19, 12, halo=2)
    rng = np.random.default_rng(5)
    fields = [rng.random(geo.shape) * 2 - 1 for _ in range(5)]
    for n, value in enumerate((np.inf, -np.inf, np.nan, 5e-324, -1e-310, 0.0, -0.0, 1e-300, 2e150, -1e-160)):
        for f in range(5):
            fields[f][2 + (n * 3 + f) % 12, 2 + (n * 7 + 2 * f) % 19, 2 + (n * 11 + 5 * f) % 40] = value
    got = _launch(cuda, fields, geo, mode, dt)
    with np.errstate(all="ignore"):
        step = api.advection_step(dict(zip("UVW", fields)), geo.dx, geo.dy, geo.dz, geo.halo, fields[3:])
        want = [step[k] for k in ("U", "V", "W", "S0", "S1")]
        if mode == native.ADVANCE:
            want = [api.euler(a.copy(), t, dt, geo.halo) for a, t in zip(fields, want)]
    for g, w in zip(got, want):
        w = w[geo.interior()]
        assert np.array_equal(np.isfinite(g), np.isfinite(w))
        ordinary = np.isfinite(w) & (np.abs(w) < 1e3)  # points without the largest value in their stencil
        assert np.abs(g[ordinary] - w[ordinary]).max() <= 1e-12 * np.abs(w[ordinary]).max()


def test_zero_and_tiny_fields(cuda):
    """Fields at rest stay exactly zero, and results below the normal range are rounded to it, not lost."""
    geo = wl.Geometry(34, 9, 5, halo=1)
    zeros = [np.zeros(geo.shape) for _ in range(4)]
    zeros[1][...] = -0.0
    for g in _launch(cuda, zeros, geo):
        assert (g == 0.0).all()
    rng = np.random.default_rng(6)
    tiny = [rng.random(geo.shape) * s for s in (1.0, 1.0, 1.0, 1e-300, 1e-312)]
    q = _velocity(tiny, geo)
    for n, (g, w) in enumerate(zip(_launch(cuda, tiny, geo), _extended(tiny, geo))):
        unit = 0.5 * float(np.abs(tiny[n]).max()) * q
        assert (np.abs(g.astype(X) - w) <= 2.0 ** -50 * np.abs(w) + 2.0 ** -49 * unit + 2 * 5e-324).all(), n
