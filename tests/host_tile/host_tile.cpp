// The advection tiles of the CUDA headers run on the host, one std::thread per
// CUDA thread: the same source, so that what a tile computes, which barriers
// its threads meet at and what depends on the chunk's depth can be checked
// without a GPU. Built and called by tests/host_tile/__init__.py.
#include <cuda_runtime.h>

#include <thread>
#include <vector>

#include "advection_fast.cuh"
#include "advection_faces.cuh"
#include "../soft_fp64/operations.h"

namespace {
using namespace f2c;

template <class F>
bool run_block(int warps, F &&body) {
    HostBlock block(32 * warps);
    std::vector<std::thread> threads;
    for (int w = 0; w < warps; ++w)
        for (int l = 0; l < 32; ++l)
            threads.emplace_back([&, w, l] {
                threadIdx = {(unsigned)l, (unsigned)w, 0};
                host_block = &block;
                body();
            });
    for (auto &t : threads) t.join();
    return !block.mixed;
}

// Every block of one launch, one after another; false when the threads of one met at different barriers.
template <int NS, int MASK>
bool launch(const AdvArgs &a, bool fast) {
    bool uniform = true;
    for (int k0 = 0; k0 < a.nz; k0 += a.kz)
        for (int y = 0; y * 8 < a.ny; ++y)
            for (int x = 0; x * 32 < a.nx; ++x) {
                const int k1 = min(k0 + a.kz, a.nz);
                if (fast) {
                    std::vector<long long> smem(FastSmem<NS, kFastTY>::bytes / 8 + 1);
                    uniform &= run_block(kFastTY, [&] { fast_tile<NS, MASK, kFastTY>(a, x, y, k0, k1, smem.data()); });
                } else {
                    std::vector<double> smem(FaceSmem<NS, MASK>::bytes / 8 + 1);
                    uniform &= run_block(kFaceTY + 1, [&] { faces_tile<NS, MASK>(a, x, y, k0, k1, smem.data()); });
                }
            }
    return uniform;
}

AdvArgs arguments(const double *const *in, double *const *out, int nscalar, const int *n, const double *d, int mode,
                  double dt, int kz) {
    AdvArgs a{};
    a.u = in[0]; a.v = in[1]; a.w = in[2];
    for (int f = 0; f < 3; ++f) a.out[f] = out[f];
    for (int f = 0; f < nscalar; ++f) {
        a.s[f] = in[3 + f];
        a.st[f] = out[3 + f];
    }
    a.nscalar = nscalar;
    a.mode = mode;
    a.dt = dt;
    a.nx = n[0]; a.ny = n[1]; a.nz = n[2]; a.h = n[3];
    a.kz = kz;
    a.sx = n[0] + 2 * n[3];
    a.plane = a.sx * (n[1] + 2 * n[3]);
    a.c = make_coefficients(d[0], d[1], d[2]);
    a.f = make_fast_coefficients(d[0], d[1], d[2], mode, dt);
    return a;
}
}  // namespace

// 0: run; 1: the threads of a block met at different barriers; 2: no such instantiation.
extern "C" int host_step(int fast, const double *const *in, double *const *out, int nscalar, const int *n,
                         const double *d, int mode, double dt, int kz) {
    const AdvArgs a = arguments(in, out, nscalar, n, d, mode, dt, kz);
    const int mask = mode == 2 ? 7 | kFillMask : (out[0] ? 1 : 0) | (out[1] ? 2 : 0) | (out[2] ? 4 : 0);
    switch (mask * 8 + nscalar) {
    case 7 * 8 + 0: return !launch<0, 7>(a, fast);
    case 7 * 8 + 1: return !launch<1, 7>(a, fast);
    case 7 * 8 + 2: return !launch<2, 7>(a, fast);
    case 15 * 8 + 1: return !launch<1, 15>(a, fast);
    case 1 * 8 + 0: return !launch<0, 1>(a, fast);
    case 1 * 8 + 1: return !launch<1, 1>(a, fast);
    case 2 * 8 + 0: return !launch<0, 2>(a, fast);
    case 2 * 8 + 1: return !launch<1, 2>(a, fast);
    case 4 * 8 + 0: return !launch<0, 4>(a, fast);
    case 4 * 8 + 1: return !launch<1, 4>(a, fast);
    case 0 * 8 + 1: return !launch<1, 0>(a, fast);
    default: return 2;
    }
}

// The fast-fp kernel's FP64 form at every point.
extern "C" void host_fp64_form(const double *const *in, double *const *out, int nscalar, const int *n, const double *d,
                               int mode, double dt) {
    const AdvArgs a = arguments(in, out, nscalar, n, d, mode, dt, 1);
    for (int k = 0; k < a.nz; ++k)
        for (int j = 0; j < a.ny; ++j)
            for (int i = 0; i < a.nx; ++i) {
                if (mode) fast_point_fp64<false, true>(a, i, j, k, ~0u);
                else fast_point_fp64<false, false>(a, i, j, k, ~0u);
            }
}

// An operation of tests/soft_fp64/operations.h on n pairs.
extern "C" void host_operations(int op, const double *a, const double *b, double *out, unsigned char *left, long long n) {
    for (long long i = 0; i < n; ++i) {
        bool l;
        out[i] = soft_cases::operation(op, a[i], b[i], l);
        left[i] = l;
    }
}
