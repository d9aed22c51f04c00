"""The work a user of this framework has it do, as cases that can be timed and checked.

Each case goes through the public entry points (``compiler.native``, the residency domain with the generated
entries, the server): the advection step in both numerical contracts, from the 64 x 64 x 32 grid of the plain
configuration to the 512 x 512 x 128 one, in every output mode, the uneven ensemble, the three generality stencils,
the step with the fields in host memory, and a serving run. A case is a dict of plain values whose ``kind`` says
which path it takes. Inputs are the recipes of ``compiler.workloads``: sums of sine modes with noise for the
velocities, uniform values and Gaussian blobs for the scalars, uniform [0, 1) with zero boundaries for the stencils.
"""

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

_PACKAGE = Path(__file__).resolve().parent.parent / "fortran-to-cuda_gb300"
if str(_PACKAGE) not in sys.path:
    sys.path.insert(0, str(_PACKAGE))

from compiler import emission, native, scheduling, serving  # noqa: E402
from compiler import workloads as wl  # noqa: E402
from compiler.resident.domain import ResidentDomain  # noqa: E402
from compiler.runtime import abi  # noqa: E402

MODES = {"tendency": native.TENDENCY, "advance": native.ADVANCE, "filled": native.ADVANCE_FILLED}
VARIANTS = {"fast": native.FAST, "strict": native.FACES}
LARGEST = 512 * 512 * 128  # points of the largest grid


def _advection(name, numerics, nx, ny, nz, nscalar, mode, halo=2, pad=0, outputs="UVW", field="modes"):
    return {"name": name, "kind": "advection", "numerics": numerics, "nx": nx, "ny": ny, "nz": nz, "halo": halo,
            "pad": pad, "nscalar": nscalar, "mode": mode, "outputs": outputs, "field": field}


def listed():
    return [
        # the plain configuration: one complete Euler step of a small grid, where the launch and its latency count
        _advection("step-small-fast", "fast", 64, 64, 32, 0, "filled"),
        # the reference driver's default: CDU alone on 64^3 with one ghost layer, uniform random fields
        _advection("cdu-small-strict", "strict", 64, 64, 64, 0, "tendency", halo=1, outputs="U", field="uniform"),
        # the headline step in both numerical contracts
        _advection("step-large-fast", "fast", 512, 512, 128, 3, "tendency"),
        _advection("step-large-strict", "strict", 512, 512, 128, 3, "tendency"),
        # ordinary single instances, ragged against every tile: a pitched Euler step, and a complete one
        _advection("step-odd-fast", "fast", 257, 193, 61, 2, "advance", pad=3),
        _advection("step-odd-strict", "strict", 161, 203, 47, 1, "filled"),
        # the uneven ensemble, one persistent launch a step, replayed as the batch's own graph
        {"name": "ensemble-fast", "kind": "ensemble", "numerics": "fast", "count": 64, "shapes": 1},
        # the generality stencils at their configured sizes
        {"name": "diffusion-large", "kind": "diffusion", "nx": 384, "ny": 384, "nz": 384, "dx": 1.0},
        {"name": "jacobi-large", "kind": "jacobi", "nx": 8192, "ny": 8192},
        {"name": "yee-large", "kind": "yee", "nx": 4096, "ny": 4096},
        # a program whose host code rewrites the inputs and reads the outputs every step, through the residency runtime
        {"name": "resident-host", "kind": "resident", "numerics": "fast", "nx": 256, "ny": 256, "nz": 128, "halo": 2,
         "nscalar": 3},
        # a serving run: jobs of the serving stream, every result kept. The stream's jobs ask for up to 100 steps;
        # here at most 8, because the smallest of these inviscid fields steepen and overflow after some 20
        {"name": "serving", "kind": "serving", "numerics": "fast", "jobs": 12, "rate": 2000.0, "stream": 5,
         "steps": 8},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["advection"] * 9 + ["ensemble"] * 3 + ["diffusion"] * 2 + ["jacobi"] * 2 + ["yee"] * 2 +
                      ["resident"] + ["serving"])
    numerics = rng.choice(["fast", "strict"])
    if kind == "advection":
        outputs = rng.choice(["UVW"] * 5 + ["U", "V", "W"])
        mode = rng.choice(list(MODES)) if outputs == "UVW" else rng.choice(["tendency", "advance"])
        return {"kind": kind, "numerics": numerics, "nx": _log(rng, 24, 512), "ny": _log(rng, 24, 512),
                "nz": _log(rng, 8, 128), "halo": rng.choice([1, 2]), "pad": rng.choice([0, 0, 3, 4]),
                "nscalar": rng.randint(0, 4 if outputs == "UVW" else 1), "mode": mode, "outputs": outputs,
                "field": rng.choice(["modes", "modes", "uniform"])}
    if kind == "ensemble":
        return {"kind": kind, "numerics": numerics, "count": _log(rng, 4, 40), "shapes": rng.randint(2, 10**6)}
    if kind == "diffusion":
        return {"kind": kind, "nx": _log(rng, 24, 384), "ny": _log(rng, 24, 384), "nz": _log(rng, 24, 384),
                "dx": rng.choice([1.0, 0.5, 0.3])}
    if kind in ("jacobi", "yee"):
        top = 8192 if kind == "jacobi" else 4096
        return {"kind": kind, "nx": _log(rng, 128, top), "ny": _log(rng, 128, top)}
    if kind == "resident":
        return {"kind": kind, "numerics": numerics, "nx": _log(rng, 48, 256), "ny": _log(rng, 48, 256),
                "nz": _log(rng, 24, 128), "halo": 2, "nscalar": rng.randint(0, 3)}
    return {"kind": kind, "numerics": numerics, "jobs": rng.randint(3, 9), "rate": rng.choice([200.0, 2000.0]),
            "stream": rng.randint(1, 10**6), "steps": rng.randint(2, 8)}


# --- inputs and the call -----------------------------------------------------------------------------


def _geometry(case):
    if case.get("field") == "uniform":  # the reference driver's spacing
        return wl.Geometry(case["nx"], case["ny"], case["nz"], case["halo"], 1.0 / case["nx"], 1.0 / case["ny"],
                           1.0 / case["nz"])
    return wl.Geometry(case["nx"], case["ny"], case["nz"], case["halo"])


def _fill(f, kind, h):
    """The boundary fill on a (nz+2h, ny+2h, nx+2h) tensor, in place."""
    return wl.fill_halo(f, kind, h)


def _inputs(case, seed):
    """U, V, W and the scalars as padded device tensors."""
    geo = _geometry(case)
    if case.get("field") == "uniform":
        g = torch.Generator(device="cuda").manual_seed(seed)
        return [torch.rand(geo.shape, generator=g, dtype=torch.float64, device="cuda")
                for _ in range(3 + case["nscalar"])]
    fields = wl.advection_fields_device(geo, seed, case["nscalar"], torch)
    return [_fill(f, 1 if n == 2 else 0, geo.halo) for n, f in enumerate(fields)]


def _pitched(fields, pad):
    if not pad:
        return fields
    out = []
    for f in fields:
        wide = torch.zeros((f.shape[0], f.shape[1], f.shape[2] + pad), dtype=torch.float64, device="cuda")
        wide[:, :, :f.shape[2]] = f
        out.append(wide)
    return out


DT = 0.1


def _dt(case):
    return 0.0 if case["mode"] == "tendency" else (DT if case["field"] == "modes" else 0.1 / max(
        case["nx"], case["ny"], case["nz"]))


def _selected(case):
    """Which of U, V, W and the scalars the case writes."""
    return [name in case["outputs"] for name in "UVW"] + [True] * case["nscalar"]


def _prepare_advection(case, seed):
    geo = _geometry(case)
    ins = _pitched(_inputs(case, seed), case["pad"])
    outs = [torch.zeros_like(t) for t in ins]
    grid = native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz, sx=ins[0].shape[2])
    return {"ins": ins, "outs": outs, "grid": grid, "mode": MODES[case["mode"]], "dt": _dt(case),
            "variant": VARIANTS[case["numerics"]], "which": _selected(case)}


def _run_advection(s):
    p = [t.data_ptr() for t in s["ins"]]
    q = [t.data_ptr() if w else None for t, w in zip(s["outs"], s["which"])]
    native.advection(s["grid"], *p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:], mode=s["mode"], dt=s["dt"],
                     stream=torch.cuda.current_stream().cuda_stream, variant=s["variant"])
    return [t for t, w in zip(s["outs"], s["which"]) if w]


def _ensemble_geometries(case):
    return [wl.Geometry(*shape) for shape in wl.ensemble_shapes(64, seed=case["shapes"])[:case["count"]]]


def _ensemble_inputs(case, seed):
    out = []
    for n, geo in enumerate(_ensemble_geometries(case)):
        f = wl.advection_fields_device(geo, 1000 * seed + n, 1, torch)
        out.append([_fill(t, 1 if m == 2 else 0, geo.halo) for m, t in enumerate(f)])
    return out


def _prepare_ensemble(case, seed):
    geometries, ins = _ensemble_geometries(case), _ensemble_inputs(case, seed)
    # every instance's U tendency in one allocation, and so on: an instance's output is a piece of each
    total = sum(math.prod(geo.shape) for geo in geometries)
    outs = [torch.zeros(total, dtype=torch.float64, device="cuda") for _ in range(4)]
    grids, fields, at = [], [], 0
    for geo, f in zip(geometries, ins):
        p, q = [t.data_ptr() for t in f], [o.data_ptr() + 8 * at for o in outs]
        grids.append(native.make_grid(geo.nx, geo.ny, geo.nz, geo.halo, geo.dx, geo.dy, geo.dz))
        fields.append(native.make_fields(*p[:3], *q[:3], scalars=p[3:], scalar_out=q[3:]))
        at += math.prod(geo.shape)
    gpu = torch.cuda.get_device_name(0)
    kz = scheduling.kz_for([(g.nx, g.ny, g.nz) for g in geometries], gpu, 1, numerics=case["numerics"])
    batch = native.Batch(grids, fields, kz=kz, tile_rows=scheduling.rows_for(gpu, 1, numerics=case["numerics"]))
    workspace = torch.empty(batch.workspace_bytes(), dtype=torch.uint8, device="cuda")
    batch.prepare(workspace.data_ptr(), workspace.numel(), torch.cuda.current_stream().cuda_stream)
    batch.set_fast_fp(case["numerics"] == "fast")
    return {"batch": batch, "workspace": workspace, "ins": ins, "outs": outs}


def _run_ensemble(s):
    s["batch"].graph_step(torch.cuda.current_stream().cuda_stream)
    return s["outs"]


def _stencils():
    lib = native.load()
    lib.f2c_diffusion7_v1.argtypes = [ctypes.POINTER(native.Grid), ctypes.c_void_p, ctypes.c_void_p, ctypes.c_double,
                                      ctypes.c_double, ctypes.c_void_p]
    lib.f2c_jacobi5_v1.argtypes = [ctypes.c_void_p] * 2 + [ctypes.c_int64] * 4 + [ctypes.c_void_p]
    lib.f2c_yee2d_v1.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int64] * 4 + [ctypes.c_double] * 2 + \
        [ctypes.c_void_p]
    return lib


def _uniform(shape, count, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for _ in range(count):
        t = torch.zeros(shape, dtype=torch.float64, device="cuda")
        inner = t[(slice(1, -1),) * len(shape)]
        inner.copy_(torch.rand(inner.shape, generator=g, dtype=torch.float64, device="cuda"))
        out.append(t)
    return out


def _plane_shape(case):
    return (case["ny"] + 2, case["nx"] + 2) if case["kind"] != "diffusion" else \
        (case["nz"] + 2, case["ny"] + 2, case["nx"] + 2)


def _prepare_stencil(case, seed):
    shape = _plane_shape(case)
    s = {"lib": _stencils(), "nx": case["nx"], "ny": case["ny"]}
    if case["kind"] == "yee":
        s["fields"] = _uniform(shape, 3, seed)
    else:
        s["in"], = _uniform(shape, 1, seed)
        s["out"] = torch.zeros_like(s["in"])
    if case["kind"] == "diffusion":
        s["grid"] = native.make_grid(case["nx"], case["ny"], case["nz"], 1, case["dx"], case["dx"], case["dx"])
        s["dt"] = 0.125 * case["dx"] ** 2
    return s


def _run_diffusion(s):
    native.check(s["lib"].f2c_diffusion7_v1(ctypes.byref(s["grid"]), s["in"].data_ptr(), s["out"].data_ptr(),
                                            s["dt"], 1.0, torch.cuda.current_stream().cuda_stream))
    return s["out"]


def _run_jacobi(s):
    native.check(s["lib"].f2c_jacobi5_v1(s["in"].data_ptr(), s["out"].data_ptr(), s["nx"], s["ny"], 1, s["nx"] + 2,
                                         torch.cuda.current_stream().cuda_stream))
    return s["out"]


CH, CE = 0.5, 0.7


def _run_yee(s):
    native.check(s["lib"].f2c_yee2d_v1(*[t.data_ptr() for t in s["fields"]], s["nx"], s["ny"], 1, s["nx"] + 2, CH, CE,
                                       torch.cuda.current_stream().cuda_stream))
    return s["fields"]


class _Resident:
    """A program's open epoch: host arrays bound in a residency domain."""

    def __init__(self, case, seed):
        self.geo = _geometry(case)
        self.ins = [t.cpu().numpy() for t in _inputs(case, seed)]
        self.outs = [np.zeros_like(a) for a in self.ins]
        lib = native.runtime()
        self.functions = emission.bind(lib)
        self.domain = ResidentDomain(lib, fast_fp=case["numerics"] == "fast")
        self.domain.begin_epoch()
        self.h_in = [self.domain.bind_real64(a) for a in self.ins]
        self.h_out = [self.domain.bind_real64(a) for a in self.outs]
        self.entry = f"advection::step{case['nscalar']}"

    def step(self):
        geo = self.geo
        self.domain.host_modify(self.h_in)
        status = emission.call(self.functions, self.entry, self.domain.context, abi.GPU,
                               [*self.h_out[:3], *self.h_in, *self.h_out[3:]], [geo.dx, geo.dy, geo.dz],
                               [geo.nx, geo.ny, geo.nz, geo.halo])
        self.domain.require(status)
        self.domain.observe(self.h_out)
        return self.outs

    def __del__(self):
        try:
            self.domain.close()
        except Exception:
            pass


def _jobs(case, seed):
    jobs = serving.poisson_jobs(case["jobs"], case["rate"], seed=case["stream"])
    for n, job in enumerate(jobs):
        job.seed = 10_000 * seed + n
        job.steps = 1 + job.steps % case["steps"]
    return jobs


def _run_serving(s):
    jobs = _jobs(s["case"], s["seed"])
    serving.Server(torch, numerics=s["case"]["numerics"], keep_results=True).run(jobs)
    return [a for job in jobs for a in job.result]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "advection":
        state = _prepare_advection(case, seed)
    elif kind == "ensemble":
        state = _prepare_ensemble(case, seed)
    elif kind == "resident":
        state = {"program": _Resident(case, seed)}
    elif kind == "serving":
        state = {"case": case, "seed": seed}
    else:
        state = _prepare_stencil(case, seed)
    state["kind"] = kind
    return state


_RUN = {"advection": _run_advection, "ensemble": _run_ensemble, "diffusion": _run_diffusion, "jacobi": _run_jacobi,
        "yee": _run_yee, "resident": lambda s: s["program"].step(), "serving": _run_serving}


def run(state):
    return _RUN[state["kind"]](state)


# --- the work of a pass ------------------------------------------------------------------------------

_MOMENTUM_FLOPS = {"UVW": 93, "U": 33, "V": 33, "W": 33}  # the reference's expressions, shared sums computed once


def _advection_work(points, nscalar, outputs, mode):
    written = len(outputs) + nscalar
    flops = _MOMENTUM_FLOPS[outputs] + (3 if nscalar else 0) + 11 * nscalar
    if mode != "tendency":
        flops += 2 * written
    return points * 8 * (3 + nscalar + written), points * flops


def work(case):
    kind = case["kind"]
    if kind == "serving":
        nbytes = flops = 0
        for job in _jobs(case, 0):
            b, f = _advection_work(job.points, job.nscalar, "UVW", "filled")
            nbytes += b * job.steps
            flops += f * job.steps
    elif kind == "ensemble":
        points = sum(g.points for g in _ensemble_geometries(case))
        nbytes, flops = _advection_work(points, 1, "UVW", "tendency")
    else:
        points = case["nx"] * case["ny"] * case.get("nz", 1)
        if kind in ("advection", "resident"):
            nbytes, flops = _advection_work(points, case["nscalar"], case.get("outputs", "UVW"),
                                            case.get("mode", "tendency"))
        else:
            per_byte, per_flop = {"diffusion": (16, 10), "jacobi": (16, 4), "yee": (48, 11)}[kind]
            nbytes, flops = points * per_byte, points * per_flop
    return {"bytes": nbytes, "flops": flops}


# --- the same results in plain torch ----------------------------------------------------------------


def _at(f, h):
    nz, ny, nx = (n - 2 * h for n in f.shape)
    return lambda i, j, k: f[h + k:h + k + nz, h + j:h + j + ny, h + i:h + i + nx]


def _tendency_u(u, v, w, dx, dy, dz):
    """The U tendency; V's and W's are the same expression with the axes' roles exchanged by the caller."""
    ax, ay, az = 0.25 / dx, 0.25 / dy, 0.25 / dz
    c = u(0, 0, 0)
    div = (ax * (u(1, 0, 0) + c) * (u(1, 0, 0) + c) - ax * (c + u(-1, 0, 0)) * (c + u(-1, 0, 0))) + \
        (ay * (u(0, 1, 0) + c) * (v(1, 0, 0) + v(0, 0, 0)) -
         ay * (c + u(0, -1, 0)) * (v(1, -1, 0) + v(0, -1, 0))) + \
        (az * (u(0, 0, 1) + c) * (w(1, 0, 0) + w(0, 0, 0)) -
         az * (c + u(0, 0, -1)) * (w(1, 0, -1) + w(0, 0, -1)))
    va = v(0, 0, 0) + v(1, 0, 0) + v(0, -1, 0) + v(1, -1, 0)
    wa = w(0, 0, 0) + w(1, 0, 0) + w(0, 0, -1) + w(1, 0, -1)
    adv = 2 * ax * (u(1, 0, 0) - u(-1, 0, 0)) * c + 0.5 * ay * (u(0, 1, 0) - u(0, -1, 0)) * va + \
        0.5 * az * (u(0, 0, 1) - u(0, 0, -1)) * wa
    return 0.5 * (-div - adv)


def _tendencies(fields, geo, which):
    u, v, w = (_at(f, geo.halo) for f in fields[:3])
    out = [None] * len(fields)
    if which[0]:
        out[0] = _tendency_u(u, v, w, geo.dx, geo.dy, geo.dz)
    if which[1]:  # x and y exchanged
        sw = [lambda i, j, k, f=f: f(j, i, k) for f in (v, u, w)]
        out[1] = _tendency_u(*sw, geo.dy, geo.dx, geo.dz)
    if which[2]:  # x and z exchanged
        sw = [lambda i, j, k, f=f: f(k, j, i) for f in (w, v, u)]
        out[2] = _tendency_u(*sw, geo.dz, geo.dy, geo.dx)
    for n, f in enumerate(fields[3:]):
        s = _at(f, geo.halo)
        c = s(0, 0, 0)
        out[3 + n] = -(0.5 / geo.dx * (u(0, 0, 0) * (s(1, 0, 0) + c) - u(-1, 0, 0) * (c + s(-1, 0, 0))) +
                       0.5 / geo.dy * (v(0, 0, 0) * (s(0, 1, 0) + c) - v(0, -1, 0) * (c + s(0, -1, 0))) +
                       0.5 / geo.dz * (w(0, 0, 0) * (s(0, 0, 1) + c) - w(0, 0, -1) * (c + s(0, 0, -1))))
    return out


def _step(fields, geo, which, mode, dt, pad=0):
    """Padded outputs of one step, as ``run`` leaves them in zeroed buffers."""
    h, out = geo.halo, []
    for n, t in enumerate(_tendencies(fields, geo, which)):
        if t is None:
            continue
        o = torch.zeros_like(fields[n])
        inner = o[geo.interior()]
        inner.copy_(t if mode == "tendency" else _at(fields[n], h)(0, 0, 0) + dt * t)
        if mode == "filled":
            _fill(o, 1 if n == 2 else 0, h)
        out.append(o)
    return _pitched(out, pad)


def exact(case, seed):
    kind = case["kind"]
    if kind == "serving":  # the jobs' first fields are the server's own single-precision draws
        return None
    if kind == "advection":
        return _step(_inputs(case, seed), _geometry(case), _selected(case), case["mode"], _dt(case), case["pad"])
    if kind == "resident":
        return [t.cpu().numpy() for t in _step(_inputs(case, seed), _geometry(case), [True] * (3 + case["nscalar"]),
                                               "tendency", 0.0)]
    if kind == "ensemble":
        steps = [_step(f, geo, [True] * 4, "tendency", 0.0)
                 for f, geo in zip(_ensemble_inputs(case, seed), _ensemble_geometries(case))]
        return [torch.cat([step[n].reshape(-1) for step in steps]) for n in range(4)]
    if kind == "yee":
        ez, hx, hy = _uniform(_plane_shape(case), 3, seed)
        i = slice(1, -1)
        hx[i, i] -= CH * (ez[2:, i] - ez[i, i])
        hy[i, i] += CH * (ez[i, 2:] - ez[i, i])
        ez[i, i] += CE * ((hy[i, i] - hy[i, :-2]) - (hx[i, i] - hx[:-2, i]))
        return [ez, hx, hy]
    f, = _uniform(_plane_shape(case), 1, seed)
    out = torch.zeros_like(f)
    if kind == "diffusion":
        s = _at(f, 1)
        c = s(0, 0, 0)
        lap = (s(-1, 0, 0) + s(1, 0, 0) + s(0, -1, 0) + s(0, 1, 0) + s(0, 0, -1) + s(0, 0, 1) - 6.0 * c) / \
            (case["dx"] * case["dx"])
        out[1:-1, 1:-1, 1:-1] = c + (0.125 * case["dx"] ** 2) * lap
    else:
        out[1:-1, 1:-1] = 0.25 * (f[1:-1, :-2] + f[1:-1, 2:] + f[:-2, 1:-1] + f[2:, 1:-1])
    return out
