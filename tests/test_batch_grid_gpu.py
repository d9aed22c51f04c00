"""The persistent grid of a batch whose items all fit on the SMs at once: one CTA per SM fewer where the items are uneven
(the last ones then go to the least loaded SMs), every item a CTA where they are even. The results are those of single
launches either way."""

import pytest

from compiler import native
from compiler import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shapes,depths,nscalar,uneven", [
    ([(128, 128, 96), (256, 64, 32)], [32, 8], 1, True),   # 192 items of 32 levels, 256 of 8
    ([(128, 128, 96), (256, 64, 32)], [32, 32], 1, False),  # 192 and 64 of 32
    ([(100, 50, 30)] * 16, [32] * 16, 0, False),
    ([(40, 20, 9)], [4], 0, False)])
def test_grid(cuda, shapes, depths, nscalar, uneven):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    grids, fields, ins, single = [], [], [], []
    for n, shape in enumerate(shapes):
        geo = wl.Geometry(*shape)
        dev = wl.advection_fields_device(geo, n, nscalar, cuda)
        outs = [[cuda.zeros_like(t) for t in dev] for _ in range(2)]
        grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz)
        p, q, r = ([t.data_ptr() for t in ts] for ts in (dev, *outs))
        native.advection(grid, *p[:3], *r[:3], scalars=p[3:], scalar_out=r[3:])
        grids.append(grid)
        fields.append(native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:]))
        ins.append(dev)
        single.append(outs)
    batch = native.Batch(grids, fields, kz=depths)
    space = cuda.empty(batch.workspace_bytes(), dtype=cuda.uint8, device="cuda")
    batch.prepare(space.data_ptr(), space.numel(), 0)
    if sms == 152:
        assert batch.plan.ctas == (2 * sms if uneven else min(3 * sms, batch.plan.items))
    batch.step(0)
    cuda.cuda.synchronize()
    for got, want in single:
        for a, b in zip(got, want):
            assert cuda.equal(a.view(cuda.int64), b.view(cuda.int64))
