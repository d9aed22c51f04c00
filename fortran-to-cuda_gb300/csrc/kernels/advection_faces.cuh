// Face-sharing z-marching advection kernel for sm_103a.
//
// GB300 executes FP64 arithmetic at about 1.6 lane-operations per clock per SM
// (measured), some 75x below its FP32 rate, so this FP64 stencil is bound by
// the FP64 pipe long before HBM. The kernel therefore performs every distinct
// operation of the reference's per-point expression trees exactly once per
// grid point:
//
//  * Each flux on a cell face appears in the expressions of the two points
//    that share the face, with the same operands in the same order (IEEE
//    addition and multiplication commute exactly), so it is computed once:
//    top faces are carried in registers up the z-march, east and north faces
//    go through shared memory to the neighbour, and a ninth "edge" warp
//    supplies the tile's west column and south row.
//  * Sums shared between the CDU, CDV and CDW trees (e.g. U(j+1)+U feeds the
//    CDU y-flux, the CDV x-flux and the CDV advective average) are computed
//    once.
//  * The final multiplication by 0.5 (benchmarks/cdu/src/cdu.f90:39) is an
//    exact exponent decrement, done on the integer pipe (with the correctly
//    rounded subnormal case handled in integer arithmetic as well).
//
// Every other operation follows the reference grouping (advection_point.cuh),
// so results are bit-identical to the oracle. All products and the advective
// forms' differences are computed on the integer pipes (soft_fp64.cuh, rounded
// exactly as DMUL and DADD), without branches: the operands that those do not
// take (zeros at the walls among them) have the thread do its half of the level
// again in FP64. A warp that starts a chunk beside zero velocities (a region at
// rest, a flow without W) takes the products they are in in FP64 from the start:
// 256 x 256 x 128 with W zero 1.77 -> 1.29 ms, at rest 1.77 -> 1.60 (a choice
// level by level cost fields without zeros 4 %). Products of zeros (a uniform flow
// has no differences) need no FP64 where the advective half is done again: uniform
// 512 x 512 x 128 without scalars 5.86 -> 5.01 ms, 100 x 80 x 40 92 -> 82 us (5.81
// ms and 90 us with 27 products on the integer pipes). So do one component's alone
// beside zeros: U without V and W, 256 x 256 x 128, 570 -> 513 us (525); with all
// three that cost fields without zeros 1 %. Operation count per point: U, V, W: 9 face sums + 18 flux
// products + 15 flux differences + 48 advective-form operations = 90; scalars: 3
// shared coefficient products + 11 per scalar. Of the 126 with three scalars 69
// are left to the FP64 pipe. Measured at 512 x 512 x 128 without and with three
// scalars: 4.83 and 7.41 ms with 27 products on the integer pipes, each with a
// branch; 4.30 and 6.47 with all 48, without; 4.12 and 6.40 with the nine
// differences as well; 4.37 and 6.99 with the nine face sums instead, 4.72 and
// 6.77 with the differences and the advecting sums (registers: 72 a thread). On
// the sine-mode fields with a Gaussian tracer: 3.95 and 6.02 ms (7.13 before;
// 7.01 with one range for momentum and scalars, whose tails then cost both; 5.93
// with the warps beside zeros apart).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "advection_kernels.cuh"
#include "device.cuh"
#include "soft_fp64.cuh"

namespace f2c {

constexpr int kFaceTX = 32;       // points per tile along x (one warp)
constexpr int kFaceTY = 8;        // compute warps per tile (points along y)
constexpr int kFaceKZ = 32;       // levels per z-chunk
constexpr int kFaceThreads = kFaceTX * (kFaceTY + 1);
// Three CTAs per SM (72 registers a thread, a few spills served by L1): 27
// warps hide the FP64, integer and shared-memory latencies. What made room for
// the third CTA is phase B reading the point's own fluxes back from the shared
// rows and its values again from L1 (ldg_again) instead of holding them in
// registers across the barrier. 512 x 512 x 128 with three scalars: 6.40 ms, at
// two CTAs 6.41; without scalars 4.13 and 4.44.
constexpr int kFaceCtasPerSM = 3;
// One component with at most a scalar needs fewer registers: four CTAs of 56. CDW alone at 512 x 512 x 128 1.47 -> 1.43
// ms, CDU at 448 x 194 x 26 111 -> 105 us, V with a scalar at 358 x 294 x 88 690 -> 661 us.
template <int NS, int MASK>
constexpr int face_ctas_per_sm() { return NS <= 1 && (MASK == 1 || MASK == 2 || MASK == 4) ? 4 : kFaceCtasPerSM; }

// Exact x * 0.5 without the FP64 pipe: for normal x the exponent field drops by
// one; for the smallest normals and subnormals the significand shifts right
// with round-half-even, which is what the correctly rounded product does.
// Infinities and NaNs are returned unchanged.
__device__ __forceinline__ double exact_half(double x) {
    const long long b = __double_as_longlong(x);
    const unsigned e = (unsigned)((unsigned long long)b >> 52) & 0x7ffu;
    const long long sign = b & (long long)0x8000000000000000ULL;
    const long long m = b & 0x001fffffffffffffLL;  // significand (with the lowest exponent bit for e == 1)
    const long long small = sign | ((m >> 1) + (m & (m >> 1) & 1));
    long long r = b - (1LL << 52);
    r = e < 2 ? small : r;
    r = e == 0x7ffu ? b : r;
    return __longlong_as_double(r);
}

// IEEE negation (the sign bit flipped, exact for every value) on the integer
// pipe. Written as inline PTX so that it stays an integer operation: a plain
// `-x`, or a sign flip written in C++, becomes a floating negation that the
// compiler issues on the FP64 pipe here (measured: three FP64 additions per
// point fewer, 2 % faster, results unchanged).
#ifdef __CUDA_ARCH__
__device__ __forceinline__ double opaque_negate(double x) {
    unsigned long long r;
    asm("xor.b64 %0, %1, 0x8000000000000000;" : "=l"(r) : "l"((unsigned long long)__double_as_longlong(x)));
    return __longlong_as_double((long long)r);
}
#else
__device__ __forceinline__ double opaque_negate(double x) { return -x; }
#endif

// Whether the high word is zero but for the sign (zero, or far below what the integer products take).
__device__ __forceinline__ bool zero_high(double x) { return ((unsigned)__double2hiint(x) << 1) == 0; }

// What a warp does in FP64 at once (faces_tile).
constexpr int kRestW = 1, kRest = 2;

// A read-only global load the compiler must issue where it stands (not merged
// with an earlier load of the same address), so that a value loaded before the
// tile's barrier need not stay in a register across it.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ double ldg_again(const double *q) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(q));
    return v;
}
#else
__device__ __forceinline__ double ldg_again(const double *q) { return *q; }
#endif

// The block's barrier inside a tile's level. A warp chooses between two copies of
// the loop over the levels (faces_tile), so that the warps of a block meet here
// from different places of the program. __syncthreads has to be one place for
// the whole block; PTX's barrier.sync is a barrier by number (0, the one that
// __syncthreads uses), which every thread of the block has to reach equally
// often, from wherever: both copies reach it once a level, and every warp of a
// block has the same levels. With one barrier outside the warps' choices, each
// phase choosing for itself, 512 x 512 x 128 with three scalars took 6.11 ms
// instead of 5.92.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ void level_barrier() { asm volatile("barrier.sync 0;" ::: "memory"); }
#else
__device__ __forceinline__ void level_barrier() { __syncthreads(); }
#endif

template <int NS, int MASK>
struct FaceSmem {
    static constexpr int NF = 3 + NS;
    // [buffer][flux][row][column]: x faces have TX+1 columns (column 0 = west edge),
    // y faces TY+1 rows (row 0 = south edge).
    static constexpr int XF = kFaceTY * (kFaceTX + 1);
    static constexpr int YF = (kFaceTY + 1) * kFaceTX;
    static constexpr size_t bytes = sizeof(double) * 2 * NF * (XF + YF);
};

// One tile: columns [tx*32, tx*32+32) x [ty*8, ty*8+8) of the interior, levels
// [k0, k1). Called by every thread of a (32, 9) block; `smem` holds
// FaceSmem<NS, MASK>::bytes. Starts and ends with the shared face buffers free.
template <int NS, int MASK>
__device__ __forceinline__ void faces_tile(const AdvArgs &a, int tile_x, int tile_y, int k0, int k1, double *smem) {
    constexpr bool DO_U = MASK & 1, DO_V = MASK & 2, DO_W = MASK & 4, FILL = (MASK & kFillMask) != 0;
    constexpr bool ONE = MASK == 1 || MASK == 2 || MASK == 4;  // velocity component
    using Smem = FaceSmem<NS, MASK>;
    constexpr int NF = Smem::NF;
    double *xface = smem;                         // [2][NF][XF]
    double *yface = smem + 2 * NF * Smem::XF;     // [2][NF][YF]

    const int lane = threadIdx.x;
    const int warp = threadIdx.y;
    const bool edge = warp == kFaceTY;
    const int i0 = tile_x * kFaceTX, j0 = tile_y * kFaceTY;
    const long long sx = a.sx, plane = a.plane;
    const double *__restrict__ U = a.u;
    const double *__restrict__ V = a.v;
    const double *__restrict__ W = a.w;
    const Coefficients c = a.c;

    // Compute threads own (i, j); the edge warp's lanes own (i0+lane, j0-1) for the south row and
    // (i0-1, j0+lane) for the west column.
    const int i = i0 + lane, j = j0 + warp;
    const bool active = !edge && i < a.nx && j < a.ny;
    const bool south_lane = edge && i < a.nx;
    const bool west_lane = edge && lane < kFaceTY && j0 + lane < a.ny;
    const int ci = edge ? i : i, cj = edge ? j0 - 1 : j;  // column of the south-row role
    long long p = (long long)(ci + a.h) + sx * (long long)(cj + a.h) + plane * (long long)(k0 + a.h);
    long long pw = (long long)(i0 - 1 + a.h) + sx * (long long)(j0 + lane + a.h) + plane * (long long)(k0 + a.h);
#define LD(A, q, di, dj, dk) __ldg((A) + (q) + (di) + (dj)*sx + (dk)*plane)

    // Top-face fluxes of the level below the current one (bottom faces), carried up the march.
    double FUzb = 0.0, FVzb = 0.0, FWzb = 0.0, ftb[NS > 0 ? NS : 1];
    bool still = false, still_w = false;  // U or V, and W, are zero here
    if (active) {
        // prologue: top faces of level k0-1
        const double Um = LD(U, p, 0, 0, -1), U0 = LD(U, p, 0, 0, 0);
        const double Vm = LD(V, p, 0, 0, -1), V0 = LD(V, p, 0, 0, 0);
        const double Wm = LD(W, p, 0, 0, -1), W0 = LD(W, p, 0, 0, 0);
        still = zero_high(U0) || zero_high(V0);
        still_w = zero_high(W0) && zero_high(Wm);
        if (DO_U) {
            const double sUz = U0 + Um;
            const double sWx = LD(W, p, 1, 0, -1) + Wm;
            FUzb = (c.Az * sUz) * sWx;
        }
        if (DO_V || DO_W) {
            const double sVz = V0 + Vm;
            const double sWy = LD(W, p, 0, 1, -1) + Wm;
            if (DO_V) FVzb = (c.Az * sVz) * sWy;
        }
        if (DO_W) {
            const double sWz = W0 + Wm;
            FWzb = (c.Az * sWz) * sWz;
        }
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            const double *__restrict__ S = a.s[n];
            ftb[n] = (c.Sz * Wm) * (LD(S, p, 0, 0, 0) + LD(S, p, 0, 0, -1));
        }
    }

    // A warp that starts beside zero velocities takes the products they are in (kRestW: W's, kRest: all) in FP64 at
    // once. Its choice for the chunk (the warps of a block choose apart: level_barrier).
    const int rest = (__any_sync(0xffffffffu, still) ? kRest : 0) | (__any_sync(0xffffffffu, still_w) ? kRestW : 0);
    int buf = 0;
    auto level = [&](const int k, auto resting) {
        constexpr bool REST = decltype(resting)::value;
        double *xf = xface + buf * NF * Smem::XF;
        double *yf = yface + buf * NF * Smem::YF;
        // ---------------- phase A: own east / north / top faces, edge faces ----------------
        double U0 = 0, Ue = 0, Un = 0, Up = 0, V0 = 0, Ve = 0, Vn = 0, Vp = 0, W0 = 0, We = 0, Wn = 0, Wp = 0;
        double sUx = 0, sVx = 0, sWx = 0, sUy = 0, sVy = 0, sWy = 0, sUz = 0, sVz = 0, sWz = 0;
        double FUx = 0, FVx = 0, FWx = 0, FUy = 0, FVy = 0, FWy = 0, FUz = 0, FVz = 0, FWz = 0;
        double S0[NS > 0 ? NS : 1], fe[NS > 0 ? NS : 1], fn[NS > 0 ? NS : 1], ft[NS > 0 ? NS : 1];
        if (active) {
            U0 = LD(U, p, 0, 0, 0); Ue = LD(U, p, 1, 0, 0); Un = LD(U, p, 0, 1, 0); Up = LD(U, p, 0, 0, 1);
            V0 = LD(V, p, 0, 0, 0); Ve = LD(V, p, 1, 0, 0); Vn = LD(V, p, 0, 1, 0); Vp = LD(V, p, 0, 0, 1);
            W0 = LD(W, p, 0, 0, 0); We = LD(W, p, 1, 0, 0); Wn = LD(W, p, 0, 1, 0); Wp = LD(W, p, 0, 0, 1);
            double se[NS > 0 ? NS : 1], sn[NS > 0 ? NS : 1], st[NS > 0 ? NS : 1];
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                const double *__restrict__ S = a.s[n];
                S0[n] = LD(S, p, 0, 0, 0);
                se[n] = LD(S, p, 1, 0, 0);
                sn[n] = LD(S, p, 0, 1, 0);
                st[n] = LD(S, p, 0, 0, 1);
            }
            if (DO_U) sUx = Ue + U0;
            if (DO_U || DO_V) sVx = Ve + V0;
            if (DO_U || DO_W) sWx = We + W0;
            if (DO_U || DO_V) sUy = Un + U0;
            if (DO_V) sVy = Vn + V0;
            if (DO_V || DO_W) sWy = Wn + W0;
            if (DO_U || DO_W) sUz = Up + U0;
            if (DO_V || DO_W) sVz = Vp + V0;
            if (DO_W) sWz = Wp + W0;
            // which: 1 the fluxes without W, 2 those with it, 3 all
            auto fluxes = [&](auto which, auto mul) {
                constexpr bool UV = decltype(which)::value & 1, WITH_W = decltype(which)::value & 2;
                if (DO_U) {
                    if (UV) FUx = mul(mul(c.Ax, sUx), sUx);
                    if (UV) FUy = mul(mul(c.Ay, sUy), sVx);
                    if (WITH_W) FUz = mul(mul(c.Az, sUz), sWx);
                }
                if (DO_V) {
                    if (UV) FVx = mul(mul(c.Ax, sVx), sUy);
                    if (UV) FVy = mul(mul(c.Ay, sVy), sVy);
                    if (WITH_W) FVz = mul(mul(c.Az, sVz), sWy);
                }
                if (DO_W && WITH_W) {
                    FWx = mul(mul(c.Ax, sWx), sUz);
                    FWy = mul(mul(c.Ay, sWy), sVz);
                    FWz = mul(mul(c.Az, sWz), sWz);
                }
            };
            auto fp64 = [](double x, double y) { return ONE ? mul_rn_left(x, y) : x * y; };
            if (REST) fluxes(std::integral_constant<int, 2>{}, fp64);
            if (REST && (rest & kRest)) {
                fluxes(std::integral_constant<int, 1>{}, fp64);
            } else {
                constexpr std::integral_constant<int, REST ? 1 : 3> which{};
                ProductRange<false> range;
                fluxes(which, [&](double x, double y) { return mul_rn_range(x, y, range); });
                if (range.left()) fluxes(which, [](double x, double y) { return mul_rn_hw(x, y); });
            }
            if (NS > 0) {
                // a scalar's own range: a tracer's zeros and tails (which WIDE takes further down) cost its own products only
                ProductRange<true> shared;
                double SxU = mul_rn_range(c.Sx, U0, shared), SyV = mul_rn_range(c.Sy, V0, shared), SzW = mul_rn_range(c.Sz, W0, shared);
                if (shared.left()) {
                    SxU = mul_rn_hw(c.Sx, U0);
                    SyV = mul_rn_hw(c.Sy, V0);
                    SzW = mul_rn_hw(c.Sz, W0);
                }
#pragma unroll
                for (int n = 0; n < NS; ++n) {
                    ProductRange<true> own;
                    const double e = se[n] + S0[n], f = sn[n] + S0[n], g = st[n] + S0[n];
                    fe[n] = mul_rn_range(SxU, e, own);
                    fn[n] = mul_rn_range(SyV, f, own);
                    ft[n] = mul_rn_range(SzW, g, own);
                    if (own.left()) {
                        fe[n] = mul_rn_hw(SxU, e);
                        fn[n] = mul_rn_hw(SyV, f);
                        ft[n] = mul_rn_hw(SzW, g);
                    }
                }
            }
            const int xo = warp * (kFaceTX + 1) + lane + 1;
            const int yo = (warp + 1) * kFaceTX + lane;
            if (DO_U) { xf[0 * Smem::XF + xo] = FUx; yf[0 * Smem::YF + yo] = FUy; }
            if (DO_V) { xf[1 * Smem::XF + xo] = FVx; yf[1 * Smem::YF + yo] = FVy; }
            if (DO_W) { xf[2 * Smem::XF + xo] = FWx; yf[2 * Smem::YF + yo] = FWy; }
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                xf[(3 + n) * Smem::XF + xo] = fe[n];
                yf[(3 + n) * Smem::YF + yo] = fn[n];
            }
        } else if (edge) {
            if (south_lane) {
                // north faces of row j0-1 (the tile's south faces)
                const double u0 = LD(U, p, 0, 0, 0), un = LD(U, p, 0, 1, 0);
                const double v0 = LD(V, p, 0, 0, 0), ve = LD(V, p, 1, 0, 0), vn = LD(V, p, 0, 1, 0);
                const double vp = LD(V, p, 0, 0, 1);
                const double w0 = LD(W, p, 0, 0, 0), wn = LD(W, p, 0, 1, 0);
                const int yo = lane;
                if (DO_U) {
                    const double s_uy = un + u0, s_vx = ve + v0;
                    yf[0 * Smem::YF + yo] = (c.Ay * s_uy) * s_vx;
                }
                if (DO_V) {
                    const double s_vy = vn + v0;
                    yf[1 * Smem::YF + yo] = (c.Ay * s_vy) * s_vy;
                }
                if (DO_W) {
                    const double s_wy = wn + w0, s_vz = vp + v0;
                    yf[2 * Smem::YF + yo] = (c.Ay * s_wy) * s_vz;
                }
                if (NS > 0) {
                    const double SyV = c.Sy * v0;
#pragma unroll
                    for (int n = 0; n < NS; ++n) {
                        const double *__restrict__ S = a.s[n];
                        yf[(3 + n) * Smem::YF + yo] = SyV * (LD(S, p, 0, 1, 0) + LD(S, p, 0, 0, 0));
                    }
                }
            }
            if (west_lane) {
                // east faces of column i0-1 (the tile's west faces), row j0+lane
                const double u0 = LD(U, pw, 0, 0, 0), ue = LD(U, pw, 1, 0, 0), un = LD(U, pw, 0, 1, 0);
                const double up = LD(U, pw, 0, 0, 1);
                const double v0 = LD(V, pw, 0, 0, 0), ve = LD(V, pw, 1, 0, 0);
                const double w0 = LD(W, pw, 0, 0, 0), we = LD(W, pw, 1, 0, 0);
                const int xo = lane * (kFaceTX + 1);
                if (DO_U) {
                    const double s_ux = ue + u0;
                    xf[0 * Smem::XF + xo] = (c.Ax * s_ux) * s_ux;
                }
                if (DO_V) {
                    const double s_vx = ve + v0, s_uy = un + u0;
                    xf[1 * Smem::XF + xo] = (c.Ax * s_vx) * s_uy;
                }
                if (DO_W) {
                    const double s_wx = we + w0, s_uz = up + u0;
                    xf[2 * Smem::XF + xo] = (c.Ax * s_wx) * s_uz;
                }
                if (NS > 0) {
                    const double SxU = c.Sx * u0;
#pragma unroll
                    for (int n = 0; n < NS; ++n) {
                        const double *__restrict__ S = a.s[n];
                        xf[(3 + n) * Smem::XF + xo] = SxU * (LD(S, pw, 1, 0, 0) + LD(S, pw, 0, 0, 0));
                    }
                }
            }
        }
        level_barrier();
        // ---------------- phase B: differences of fluxes and the advective forms ----------------
        if (active) {
            const int xw = warp * (kFaceTX + 1) + lane;
            const int ys = warp * kFaceTX + lane;
            // this point's own east / north fluxes are read back from the shared rows and its values again
            // from memory (L1), rather than held in registers across the barrier
            const int xo = xw + 1, yo = ys + kFaceTX;
#define LDA(A, di, dj, dk) ldg_again((A) + p + (di) + (dj)*sx + (dk)*plane)
            const double Uc = LDA(U, 0, 0, 0), Vc = LDA(V, 0, 0, 0), Wc = LDA(W, 0, 0, 0);  // the point's own values
            const double Uw = LD(U, p, -1, 0, 0), Us = LD(U, p, 0, -1, 0), Um = LD(U, p, 0, 0, -1);
            const double Vw = LD(V, p, -1, 0, 0), Vs = LD(V, p, 0, -1, 0), Vm = LD(V, p, 0, 0, -1);
            const double Ww = LD(W, p, -1, 0, 0), Ws = LD(W, p, 0, -1, 0), Wm = LD(W, p, 0, 0, -1);
            double aU[3] = {0, 0, 0}, aV[3] = {0, 0, 0}, aW[3] = {0, 0, 0};  // the advective forms' terms
            auto advective = [&](auto which, auto mul, auto sub) {
                constexpr bool UV = decltype(which)::value & 1, WITH_W = decltype(which)::value & 2;
                if (DO_U) {
                    if (UV) aU[0] = mul(mul(c.Bux, sub(LDA(U, 1, 0, 0), Uw)), Uc);
                    if (UV) aU[1] = mul(mul(c.Buy, sub(LDA(U, 0, 1, 0), Us)), (sVx + Vs) + LD(V, p, 1, -1, 0));
                    if (WITH_W) aU[2] = mul(mul(c.Buz, sub(LDA(U, 0, 0, 1), Um)), (sWx + Wm) + LD(W, p, 1, 0, -1));
                }
                if (DO_V) {
                    if (UV) aV[0] = mul(mul(c.Bvx, sub(LDA(V, 1, 0, 0), Vw)), (sUy + Uw) + LD(U, p, -1, 1, 0));
                    if (UV) aV[1] = mul(mul(c.Bvy, sub(LDA(V, 0, 1, 0), Vs)), Vc);
                    if (WITH_W) aV[2] = mul(mul(c.Bvz, sub(LDA(V, 0, 0, 1), Vm)), (sWy + Wm) + LD(W, p, 0, 1, -1));
                }
                if (DO_W && WITH_W) {
                    aW[0] = mul(mul(c.Bwx, sub(LDA(W, 1, 0, 0), Ww)), (sUz + Uw) + LD(U, p, -1, 0, 1));
                    aW[1] = mul(mul(c.Bwy, sub(LDA(W, 0, 1, 0), Ws)), (sVz + Vs) + LD(V, p, 0, -1, 1));
                    aW[2] = mul(mul(c.Bwz, sub(LDA(W, 0, 0, 1), Wm)), Wc);
                }
            };
            auto fp64 = [](double x, double y) { return ONE ? mul_rn_left(x, y) : x * y; };
            auto difference = [](double x, double y) { return x - y; };
            if (REST) advective(std::integral_constant<int, 2>{}, fp64, difference);
            if (REST && (rest & kRest)) {
                advective(std::integral_constant<int, 1>{}, fp64, difference);
            } else {
                constexpr std::integral_constant<int, REST ? 1 : 3> which{};
                ProductRange<false> range;
                SumRange sums;
                advective(which, [&](double x, double y) { return mul_rn_range(x, y, range); },
                          [&](double x, double y) { return add_rn_range(x, opaque_negate(y), sums); });
                if (range.left() || sums.left())
                    advective(which, [](double x, double y) { return mul_rn_again(x, y); }, difference);
            }
            if (DO_U) {
                const double r = opaque_negate(((xf[0 * Smem::XF + xo] - xf[0 * Smem::XF + xw]) + (yf[0 * Smem::YF + yo] - yf[0 * Smem::YF + ys])) + (FUz - FUzb));
                if (a.out[0]) store_point_t<FILL>(a.out[0], U, p, exact_half(r - ((aU[0] + aU[1]) + aU[2])), a, 0, i, j, k);
                FUzb = FUz;
            }
            if (DO_V) {
                const double r = opaque_negate(((yf[1 * Smem::YF + yo] - yf[1 * Smem::YF + ys]) + (xf[1 * Smem::XF + xo] - xf[1 * Smem::XF + xw])) + (FVz - FVzb));
                if (a.out[1]) store_point_t<FILL>(a.out[1], V, p, exact_half(r - ((aV[0] + aV[1]) + aV[2])), a, 0, i, j, k);
                FVzb = FVz;
            }
            if (DO_W) {
                const double r = opaque_negate(((FWz - FWzb) + (yf[2 * Smem::YF + yo] - yf[2 * Smem::YF + ys])) + (xf[2 * Smem::XF + xo] - xf[2 * Smem::XF + xw]));
                if (a.out[2]) store_point_t<FILL>(a.out[2], W, p, exact_half(r - ((aW[0] + aW[1]) + aW[2])), a, 1, i, j, k);
                FWzb = FWz;
            }
#pragma unroll
            for (int n = 0; n < NS; ++n) {
                const double st = opaque_negate(((xf[(3 + n) * Smem::XF + xo] - xf[(3 + n) * Smem::XF + xw]) + (yf[(3 + n) * Smem::YF + yo] - yf[(3 + n) * Smem::YF + ys])) +
                                    (ft[n] - ftb[n]));
                if (a.st[n]) store_point_t<FILL>(a.st[n], a.s[n], p, st, a, 0, i, j, k);
                ftb[n] = ft[n];
            }
#undef LDA
        }
    };
    if (rest) {
        for (int k = k0; k < k1; ++k, p += plane, pw += plane, buf ^= 1) level(k, std::true_type{});
    } else {
        for (int k = k0; k < k1; ++k, p += plane, pw += plane, buf ^= 1) level(k, std::false_type{});
    }
#undef LD
}

#ifdef __CUDACC__
template <int NS, int MASK>
__global__ void __launch_bounds__(kFaceThreads, face_ctas_per_sm<NS, MASK>()) advection_faces_kernel(const AdvArgs a) {
    extern __shared__ double smem[];
    const int k0 = blockIdx.z * a.kz;
    faces_tile<NS, MASK>(a, blockIdx.x, blockIdx.y, k0, min(k0 + a.kz, a.nz), smem);
}
#endif

// Depth of the z-chunks of one launch: the one with the least time on the SM
// with the most CTAs, whose levels (and about half a level for a chunk's start)
// the FP64 pipe takes one after another; one CTA more is counted because the
// last ones have the SM to themselves and wait on latencies. 161 x 203 x 47 with
// a scalar: 4 levels, 0.31 ms (13, as four CTAs per SM would have, 0.35);
// 64^3, U alone: one level, 18.6 us (2: 20.5).
inline int chunk_depth(int nx, int ny, int nz) {
    const long long sms = current_sm_count();
    const long long tiles = (long long)((nx + kFaceTX - 1) / kFaceTX) * ((ny + kFaceTY - 1) / kFaceTY);
    long long best = -1;
    int depth = 1;
    for (int kz = 1; kz <= kFaceKZ && kz <= nz; ++kz) {
        const long long ctas = tiles * ((nz + kz - 1) / kz);
        const long long cost = ((ctas + sms - 1) / sms + 1) * (2 * kz + 1);
        if (best < 0 || cost <= best) {
            best = cost;
            depth = kz;
        }
    }
    return depth;
}

#ifdef __CUDACC__
template <int NS, int MASK>
cudaError_t launch_faces(const AdvArgs &a, cudaStream_t stream) {
    using Smem = FaceSmem<NS, MASK>;
    static std::atomic<unsigned long long> configured{0};
    const cudaError_t e =
        configure_shared_once(configured, (const void *)advection_faces_kernel<NS, MASK>, (int)Smem::bytes);
    if (e != cudaSuccess) return e;
    AdvArgs b = a;
    if (b.kz <= 0) b.kz = chunk_depth(b.nx, b.ny, b.nz);
    const dim3 block(kFaceTX, kFaceTY + 1, 1);
    const dim3 grid((b.nx + kFaceTX - 1) / kFaceTX, (b.ny + kFaceTY - 1) / kFaceTY, (b.nz + b.kz - 1) / b.kz);
    advection_faces_kernel<NS, MASK><<<grid, block, Smem::bytes, stream>>>(b);
    return cudaGetLastError();
}
#endif

} // namespace f2c
