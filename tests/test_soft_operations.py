"""The operations of soft_fp64.cuh that the kernels call, against IEEE arithmetic: bit for bit where they take their
operands, which is exactly where they say. Pairs of special values, signed zeros and both ends of the exponent range,
and random ones of near and far exponents that cancel, tie and round; on the host, and the shipped code on the GPU."""

import ctypes
import shutil
import subprocess

import numpy as np
import pytest

import host_tile
from test_soft_fp64 import HERE, KERNELS

OPERATIONS = {"product": 0, "wide product": 1, "sum": 2, "product again": 3, "sum again": 4}
SPECIAL = [0.0, 5e-324, 1e-310, 2.0**-1022, 2.0**-959, 2.0**-512, 2.0**-511, 0.1, 0.75, 1.0, 1.0 + 2.0**-52, 1.5, 3.0,
           2.0**53 - 1, 2.0**511, 2.0**512, 2.0**944, 2.0**945, 1e300, np.finfo(float).max, np.inf, np.nan]


def _pairs():
    special = np.array(SPECIAL + [-x for x in SPECIAL])
    a, b = (m.reshape(-1) for m in np.meshgrid(special, special))
    rng = np.random.default_rng(12)
    n = 200000
    x = (rng.random(n) + 1) * 2.0 ** rng.integers(-40, 40, n) * rng.choice([-1, 1], n)
    near = np.where(rng.random(n) < 0.5, x * (1 + rng.integers(-3, 4, n) * 2.0**-52), rng.permutation(x))
    short = np.ldexp(rng.integers(1, 1 << 27, n).astype(float), rng.integers(-30, 30, n))  # products and sums that tie
    return np.concatenate([a, x, short]), np.concatenate([b, -near, rng.permutation(short)])


def _exponent(x):
    return (x.view(np.int64) >> 52) & 0x7FF


def _check(op, a, b, got, left):
    with np.errstate(all="ignore"):
        want = a + b if op in (2, 4) else a * b
    ea, eb = _exponent(a), _exponent(b)
    if op == 0:
        may = (ea < 512) | (ea > 1534) | (eb < 512) | (eb > 1534)
    elif op == 1:
        may = (ea == 0) | (eb == 0) | (ea == 0x7FF) | (eb == 0x7FF) | (ea + eb < 1024) | (ea + eb >= 1024 + 2044)
    elif op == 2:
        least = np.minimum(ea, eb)
        may = (np.abs(ea - eb) > 31) | (least < 64) | (least > 1968) | (want == 0)
    else:
        may = np.zeros(a.shape, bool)
    assert np.array_equal(left.astype(bool), may)
    same = (got.view(np.int64) == want.view(np.int64)) | (np.isnan(got) & np.isnan(want))
    assert same[~may].all(), [(x, y) for x, y in zip(a[~may & ~same][:4], b[~may & ~same][:4])]


@pytest.mark.parametrize("name", OPERATIONS)
def test_on_the_host(name):
    a, b = _pairs()
    out, left = np.empty_like(a), np.empty(a.shape, np.uint8)
    host_tile.library().host_operations(OPERATIONS[name], *(ctypes.c_void_p(t.ctypes.data) for t in (a, b, out, left)),
                                        ctypes.c_longlong(a.size))
    _check(OPERATIONS[name], a, b, out, left)


@pytest.mark.gpu
def test_on_the_gpu(cuda, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    lib = tmp_path / "operations.so"
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared", "--fmad=false",
                    "-Xcompiler", "-fPIC", f"-I{KERNELS}", f"-I{HERE}", str(HERE / "operations_device.cu"),
                    "-o", str(lib)], check=True)
    run = ctypes.CDLL(str(lib)).soft_operations_device
    a, b = _pairs()
    da, db = cuda.from_numpy(a).cuda(), cuda.from_numpy(b).cuda()
    for op in OPERATIONS.values():
        out, left = cuda.empty_like(da), cuda.empty(a.size, dtype=cuda.uint8, device="cuda")
        assert run(op, *(ctypes.c_void_p(t.data_ptr()) for t in (da, db, out, left)), ctypes.c_longlong(a.size)) == 0
        _check(op, a, b, out.cpu().numpy(), left.cpu().numpy())
