// Factored ("fast-fp") z-marching advection kernel for sm_103a.
//
// The reference's --fast-fp build (compiler/resident/build.py:22,66-67) trades
// the strict contract for FMA contraction. This kernel computes the same
// tendencies as the strict face-sharing kernel (advection_faces.cuh) through an
// algebraically regrouped form, on the integer pipes. GB300 issues FP64 at 1.68
// lane operations per clock per SM, 64-bit integer additions and 32 x 32 + 64
// multiplications at 64 each, so what costs a thread one FP64 operation pays for
// some forty integer ones: sums and products of a point's stencil are taken in
// 64-bit fixed point at the point's own scale (wide_int.cuh), and FP64 converts
// and scales each result, two operations per field instead of some twenty.
//
// Regrouping (exact in real arithmetic; A = 0.25/d per direction). For the U
// component of benchmarks/cdu/src/cdu.f90:66-71,96-101 with the final
// multiplication by one half (:39):
//   x: Ax[(Ue+U0)^2 - (U0+Uw)^2] + 2Ax(Ue-Uw)U0 = Ax (Ue-Uw)(Ue+Uw+4U0)
//   y: Ay[n vn - s vs] + (Ay/2)(n-s)(vn+vs)
//        = (Ay/2)[2(n-s)(vn+vs) + (n+s)(vn-vs)]
// where n, s are U's north and south face sums (U(j+1)+U, U+U(j-1)) and vn, vs
// the V face sums at the same corners (V(i+1)+V at rows j and j-1); z is the y
// form with U's top/bottom face sums and W's. The advective coefficients of the
// reference (0.5/d along the component, 0.125/d across) are exactly 2A and A/2,
// and Un-Us = n-s, so the flux and advective forms share every sum. V and W
// rotate the roles (compiler/tests/fixtures/stencils/{cvd,cdw}.f90:61-66,
// 89-94). A component is the sum over the directions, each in units of its
// coefficient over x's, times one coefficient; so is a scalar with its six faces
// (advection_point.cuh).
//
// Precision: a field's values at a point's stencil keep 60 bits below the
// largest of them (an FP64 operation 53 below its own operands). Each direction
// is summed at the scale of its own factors, and brought to the largest of the
// three: along the component that is its difference's scale (a nearly uniform
// wind's is small), across it the crossing velocity's. A result is off by its two
// final roundings and 2^-56 or so of that, whatever the tile. Summed at one
// scale, the largest velocity's, a wind of 10 lost a digit for each factor of ten
// between it and a cross flow below 1e-2 (1.7e-11 of the maximum at 1e-6; the
// FP64 form 2e-16). Against exact sums the errors (2-norm) are 0.1 to 1.1 of the
// FP64 form's over the workloads' fields, uniform and nearly uniform winds,
// jets, vortices and random exponents, but where both are at the two final
// roundings (1.5e-16). What the integers cannot take (infinities, NaN, a value
// beside the point's own factors that is far larger than they are) goes to FP64
// point by point.
//
// Each value is unpacked once, by the thread that owns its cell (the frame's by
// the threads in turn), and read by its neighbours from shared memory. Values
// two levels up are already on their way by asynchronous copies: held in
// registers across the barrier instead, the loads cost 18-24 % of the step.
// 8 warps of 128 registers, two CTAs per SM; with three (80 registers, spills)
// 512 x 512 x 128 with three scalars took 1.79 ms instead of 1.54, 4-row tiles
// 2.1, 16-row tiles 2.1 (each with its frame's share of the unpacking).
// 512 x 512 x 128 with three scalars: 1.55 ms (the FP64 form 3.95); without
// scalars 0.94; 257 x 193 x 61 with two, advanced: 162 us (475); 64 instances
// with one scalar in one batched launch: 3.57 ms (9.44; 3.38 with one scale for
// all directions, which lost digits). Spacings with no power-of-two ratio: 1.71 ms
// at the first of these.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "advection_faces.cuh"
#include "advection_kernels.cuh"
#include "wide_int.cuh"

namespace f2c {

constexpr int kFastTX = 32;        // points per tile along x (one warp)
constexpr int kFastKZ = 32;        // levels per z-chunk for large grids
constexpr int kFastPrologue = 3;   // cost of a chunk's start, in half levels

// Shared memory of a tile: the wide values (wide_int.cuh) of the tile's cells
// and a one-cell frame, one plane per field and level in a ring of three levels
// (the one below, of which a thread reads only its own cell; the level; the one
// above it, being written), significands and exponents apart; and the FP64
// values on their way from global memory, two levels of them, each read only by
// the thread that asked for it.
template <int NS, int TY>
struct FastSmem {
    static constexpr int PITCH = kFastTX + 2, PLANE = (TY + 2) * PITCH;
    static constexpr int FIELDS = 3 + NS;
    static constexpr int FRAME = 2 * kFastTX + 2 * TY + 2;  // cells of the frame the stencils reach
    static constexpr int THREADS = kFastTX * TY;
    static constexpr int TURNS = (FIELDS * FRAME + THREADS - 1) / THREADS;
    static constexpr int LEVEL = FIELDS * PLANE;
    static constexpr int AHEAD = (FIELDS + TURNS) * THREADS;  // values on their way, a level
    static constexpr int bytes = 8 * (3 * LEVEL + 2 * AHEAD) + 2 * 3 * LEVEL;
};

template <int TY>
constexpr int fast_threads() { return kFastTX * TY; }

// CTAs per SM a tile height is compiled for: 16 warps of 128 registers. (Shared memory allows them but for tiles of 4
// rows with three or four scalars, 57 and 67 KB a CTA, of which three fit.)
template <int TY>
constexpr int fast_ctas_per_sm() { return TY <= 4 ? 4 : (TY <= 8 ? 2 : 1); }

// Exponents above the values that a component reads itself at which it still keeps as many bits as FP64: 60 - 5 of them.
constexpr int kWideSlack = 5;

constexpr int kFastTY = 8;  // tile height of the single-instance launches

// One momentum component in FP64 straight from memory. P is the component, d1
// the stride along it; Q and R are the two other velocities, d2 and d3 the
// strides along those. With n, s the component's face sums across an axis and
// vn, vs the crossing velocity's, a direction is n(3vn+vs) - s(3vs+vn); along
// the component (f1-f0)(f1+f0+4c).
static __device__ double fast_component_fp64(const double *P, const double *Q, const double *R, long long d1,
                                             long long d2, long long d3, double g, double c2, double c3,
                                             double start) {
    const double c = P[0];
    auto cross = [&](const double *F, long long d) {
        const double p = P[d] + c, pn = c + P[-d], q = F[d1] + F[0], qn = F[d1 - d] + F[-d];
        return __fma_rn(p, __fma_rn(3.0, q, qn), -(pn * __fma_rn(3.0, qn, q)));
    };
    const double f1 = P[d1], f0 = P[-d1];
    double t = __fma_rn(c3, cross(R, d3), start);
    t = __fma_rn(c2, cross(Q, d2), t);
    return __fma_rn(g, (f1 - f0) * __fma_rn(4.0, c, f1 + f0), t);
}

// The fields of `which` (bit n: U, V, W, scalars) at one point in FP64, for the
// points whose stencil the wide integers cannot take (infinities, NaN,
// subnormals, results near the ends of the exponent range) and for grids whose
// coefficients they cannot. One call for a point: a call in each field's way
// cost 10 % of the step.
template <bool FILL, bool ADVANCE>
static __device__ __noinline__ void fast_point_fp64(const AdvArgs &a, int i, int j, int k, unsigned which) {
    const long long sx = a.sx, plane = a.plane;
    const long long p = (long long)(i + a.h) + sx * (long long)(j + a.h) + plane * (long long)(k + a.h);
    const double *U = a.u + p, *V = a.v + p, *W = a.w + p;
    const FastCoefficients &c = a.f;
    for (int f = 0; f < 3 + a.nscalar; ++f) {
        double *out = f < 3 ? a.out[f] : a.st[f - 3];
        if (!(which >> f & 1) || !out) continue;
        const double *S = (f == 0 ? a.u : (f == 1 ? a.v : (f == 2 ? a.w : a.s[f - 3]))) + p;
        const double start = ADVANCE ? S[0] : 0.0;
        double t;
        if (f == 0) {
            t = fast_component_fp64(U, V, W, 1, sx, plane, c.gx, c.cy, c.cz, start);
        } else if (f == 1) {
            t = fast_component_fp64(V, U, W, sx, 1, plane, c.gy, c.cx, c.cz, start);
        } else if (f == 2) {
            t = fast_component_fp64(W, U, V, plane, 1, sx, c.gz, c.cx, c.cy, start);
        } else {
            const double e = c.sx * U[0], w = c.sx * U[-1], n = c.sy * V[0], s = c.sy * V[-sx], u = c.sz * W[0],
                         b = c.sz * W[-plane];
            t = __fma_rn(S[0], ((w - e) + (s - n)) + (b - u), start);
            t = __fma_rn(-e, S[1], t);
            t = __fma_rn(w, S[-1], t);
            t = __fma_rn(-n, S[sx], t);
            t = __fma_rn(s, S[-sx], t);
            t = __fma_rn(-u, S[plane], t);
            t = __fma_rn(b, S[-plane], t);
        }
        if (FILL) store_filled(out, f == 2 ? 1 : 0, a, i, j, k, t);
        else out[p] = t;
    }
}

#ifdef __CUDA_ARCH__
// An 8-byte copy from global to shared memory that runs on while the thread does (cp.async).
__device__ __forceinline__ void fetch(long long *to, const double *from) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
#else
__device__ __forceinline__ void fetch(long long *to, const double *from) { *to = __double_as_longlong(*from); }
__device__ __forceinline__ void fetch_commit() {}
template <int N>
__device__ __forceinline__ void fetch_wait() {}
#endif

// One tile: columns [tile_x*32, +32) x [tile_y*TY, +TY) of the interior, levels
// [k0, k1), for one output mode (ADVANCE: forward Euler, else the tendency).
// Called by every thread of a (32, TY) block; `smem` holds
// FastSmem<NS, TY>::bytes. Starts with the buffers free; a caller that goes on to
// another tile has a barrier in between.
template <int NS, int MASK, int TY, bool ADVANCE, bool SCALED>
__device__ __forceinline__ void fast_tile_mode(const AdvArgs &a, int tile_x, int tile_y, int k0, int k1,
                                               long long *smem) {
    constexpr bool DU = MASK & 1, DV = (MASK >> 1) & 1, DW = (MASK >> 2) & 1;
    constexpr bool filled = (MASK & kFillMask) != 0;  // F2C_ADVANCE_FILLED: outputs with their ghost images
    using Sm = FastSmem<NS, TY>;
    constexpr int PITCH = Sm::PITCH, PLANE = Sm::PLANE, LEVEL = Sm::LEVEL, FIELDS = Sm::FIELDS;
    const int lane = threadIdx.x;
    const int warp = threadIdx.y;
    const int i0 = tile_x * kFastTX, j0 = tile_y * TY;
    const int i = i0 + lane, j = j0 + warp;
    const bool active = i < a.nx && j < a.ny;
    const bool inside = i <= a.nx && j <= a.ny;  // cells the stencils reach
    const bool across = i < a.h || i >= a.nx - a.h || j < a.h || j >= a.ny - a.h;
    const long long sx = a.sx, plane = a.plane;
    const FastCoefficients &c = a.f;
    long long *const ring = smem;
    long long *const ahead = smem + 3 * LEVEL + warp * kFastTX + lane;  // this thread's values on their way
    short *const ring_e = reinterpret_cast<short *>(smem + 3 * LEVEL + 2 * Sm::AHEAD);
    auto field = [&](int f) { return f == 0 ? a.u : (f == 1 ? a.v : (f == 2 ? a.w : a.s[f - 3])); };
    auto put = [&](int at, double x) {
        const Wide w = wide_pack(x);
        ring[at] = w.m;
        ring_e[at] = (short)w.e;
    };

    // The frame around the tile (the rows south and north of it, its west and east columns, the corners U
    // north-west and V south-east): one value of one field to each of the first FIELDS * FRAME turns of the threads.
    constexpr int TURNS = Sm::TURNS;
    const double *frame_at[TURNS];
    int frame_to[TURNS];
#pragma unroll
    for (int t = 0; t < TURNS; ++t) {
        const int n = t * kFastTX * TY + warp * kFastTX + lane;
        const int f = n / Sm::FRAME, m = n - f * Sm::FRAME;
        const int r = m - 2 * kFastTX;
        const int row = m < kFastTX ? -1 : (r < 0 ? TY : (r < TY ? r : (r < 2 * TY ? r - TY : (r == 2 * TY ? TY : -1))));
        const int col = r < 0 ? (m & (kFastTX - 1)) : (r < TY || r == 2 * TY ? -1 : kFastTX);
        const bool use = f < FIELDS && i0 + col <= a.nx && j0 + row <= a.ny;
        const double *base = a.u;
#pragma unroll
        for (int g = 1; g < FIELDS; ++g)
            if (f == g) base = field(g);
        frame_at[t] = base + (i0 + col + a.h) + sx * (long long)(j0 + row + a.h) + plane * (long long)(k0 - 1 + a.h);
        frame_to[t] = use ? f * PLANE + (row + 1) * PITCH + col + 1 : -1;
    }
    const int own = (warp + 1) * PITCH + lane + 1;
    const long long p0 = (long long)(i + a.h) + sx * (long long)(j + a.h) + plane * (long long)(k0 + a.h);
    long long p = p0;
    // the values of level k (offset `at` from level k0's), into half `half` of the buffer
    auto fetch_level = [&](long long *to, long long at, long long frame_step) {
        if (inside) {
#pragma unroll
            for (int f = 0; f < FIELDS; ++f) fetch(to + f * Sm::THREADS, field(f) + at);
        }
#pragma unroll
        for (int t = 0; t < TURNS; ++t) {
            if (frame_to[t] >= 0) {
                fetch(to + (FIELDS + t) * Sm::THREADS, frame_at[t]);
                frame_at[t] += frame_step;
            }
        }
        fetch_commit();
    };
    auto put_level = [&](const long long *from, int to) {
        if (inside) {
#pragma unroll
            for (int f = 0; f < FIELDS; ++f) put(to + f * PLANE + own, __longlong_as_double(from[f * Sm::THREADS]));
        }
#pragma unroll
        for (int t = 0; t < TURNS; ++t) {
            if (frame_to[t] >= 0) put(to + frame_to[t], __longlong_as_double(from[(FIELDS + t) * Sm::THREADS]));
        }
    };
    // levels k0-1 (slot 2: own column, and W's frame) and k0 (slot 0); level k0+1 on its way
    Wide wem{0, 0}, wnm{0, 0};  // W east and north of the column a level down (U and V read them): carried up
    fetch_level(ahead, p - plane, plane);
    fetch_level(ahead + Sm::AHEAD, p, plane);
    fetch_wait<1>();
    put_level(ahead, 2 * LEVEL);
    fetch_level(ahead, p + plane, plane);
    fetch_wait<1>();
    put_level(ahead + Sm::AHEAD, 0);
    if (DU || DV) {
        __syncthreads();
        const int n = 2 * LEVEL + 2 * PLANE + own;
        wem = {ring[n + 1], ring_e[n + 1]};
        wnm = {ring[n + PITCH], ring_e[n + PITCH]};
    }

    int below = 2, slot = 0;  // ring slots of levels k-1 and k
    int half = 0;             // of the buffer, with level k+1
    for (int k = k0; k < k1; ++k, p += plane, half ^= 1) {
        const int above = 3 - below - slot;
        // level k+2 on its way, and level k+1 into the ring
        if (k + 1 < k1) fetch_level(ahead + (half ^ 1) * Sm::AHEAD, p + 2 * plane, plane);
        else fetch_commit();
        fetch_wait<1>();
        put_level(ahead + half * Sm::AHEAD, above * LEVEL);
        double old[ADVANCE ? FIELDS : 1];  // the fields' values, asked for ahead of their use
        if (ADVANCE && active) {
#pragma unroll
            for (int f = 0; f < FIELDS; ++f) old[f] = ldg_again(field(f) + p);
        }
        __syncthreads();
        if (active) {
            const long long *now = ring + slot * LEVEL + own, *next = ring + above * LEVEL + own,
                            *prev = ring + below * LEVEL + own;
            const short *now_e = ring_e + slot * LEVEL + own, *next_e = ring_e + above * LEVEL + own,
                      *prev_e = ring_e + below * LEVEL + own;
            auto at = [&](int f, int row, int col) {
                const int n = f * PLANE + row * PITCH + col;
                return Wide{now[n], now_e[n]};
            };
            auto over = [&](int f, int row, int col) {
                const int n = f * PLANE + row * PITCH + col;
                return Wide{next[n], next_e[n]};
            };
            auto under = [&](int f) { return Wide{prev[f * PLANE], prev_e[f * PLANE]}; };
            unsigned slow = 0;  // the fields to be done again in FP64
            // whether the new value has ghost images (store_filled), or is a W wall face
            const bool images = filled && (across || k < a.h || k >= a.nz - 1 - a.h);
            // a component's or scalar's value from its sum T at exponent e, stored
            auto finish = [&](int f, long long T, int e) {
                const int g = f < 3 ? 0 : 1;
                double *o = f < 3 ? a.out[f] : a.st[f - 3];
                bool fits;
                const double t = wide_result<ADVANCE>(T, e, c.wide_hi[g], c.wide_lo[g], c.wide_e[g],
                                                      ADVANCE ? old[ADVANCE ? f : 0] : 0.0, fits);
                if (!fits) slow |= 1u << f;
                if (!o) return;
                if (images) store_filled(o, f == 2 ? 1 : 0, a, i, j, k, t);
                else o[p] = t;
            };
            const Wide z{0, 0};
            // the stencil of U, V and W, each field aligned to its own largest exponent in it
            const Wide u0 = at(0, 0, 0), v0 = at(1, 0, 0), w0 = at(2, 0, 0);
            const Wide uw = at(0, 0, -1), un = DU || DV ? at(0, 1, 0) : z, up = DU || DW ? over(0, 0, 0) : z;
            const Wide ue = DU ? at(0, 0, 1) : z, us = DU ? at(0, -1, 0) : z, um = DU ? under(0) : z;
            const Wide uwn = DV ? at(0, 1, -1) : z, uwp = DW ? over(0, 0, -1) : z;
            const Wide vs = at(1, -1, 0), ve = DU || DV ? at(1, 0, 1) : z, vp = DV || DW ? over(1, 0, 0) : z;
            const Wide vn = DV ? at(1, 1, 0) : z, vw = DV ? at(1, 0, -1) : z, vm = DV ? under(1) : z;
            const Wide ves = DU ? at(1, -1, 1) : z, vsp = DW ? over(1, -1, 0) : z;
            const Wide wm = under(2), we = DU || DV || DW ? at(2, 0, 1) : z, wn = DU || DV || DW ? at(2, 1, 0) : z;
            const Wide ww = DW ? at(2, 0, -1) : z, ws = DW ? at(2, -1, 0) : z, wp = DW ? over(2, 0, 0) : z;
            // (pu, pv, pw: over what the component reads of itself)
            const int pu = max3(max3(u0.e, uw.e, up.e), max3(un.e, ue.e, us.e), um.e), EU = max3(pu, uwn.e, uwp.e);
            const int pv = max3(max3(v0.e, vs.e, vp.e), max3(vn.e, ve.e, vw.e), vm.e), EV = max3(pv, ves.e, vsp.e);
            const int pw = max3(max3(w0.e, wm.e, wp.e), max3(wn.e, we.e, ww.e), ws.e), EW = DU || DV ? max3(pw, wem.e, wnm.e) : pw;
            const int tu = EU + 3, tv = EV + 3, tw = EW + 3;
            const long long au0 = wide_align(u0, tu), auw = wide_align(uw, tu), aun = wide_align(un, tu),
                            aup = wide_align(up, tu);
            const long long av0 = wide_align(v0, tv), avs = wide_align(vs, tv), ave = wide_align(ve, tv),
                            avp = wide_align(vp, tv);
            const long long aw0 = wide_align(w0, tw), awm = wide_align(wm, tw), awe = wide_align(we, tw),
                            awn = wide_align(wn, tw);
            const int ux = max(u0.e, uw.e), vx = max(v0.e, vs.e), wx = max(w0.e, wm.e);  // of the faces at the point
            // a component P's three sums brought to the largest of their scales: along its own axis (A, lifted by n bits)
            // and across the two others; FP, F2 and F3 are the exponents of P and of the velocities across, in units of
            // the directions' coefficients over x's; p, p2 and p3 those of the values that P's own sums read. A sum whose
            // scale lies above those (next to a far larger value that another component reads) is left to FP64. (One
            // test for the three components sent all three there beside a wall: 64 x 64 x 32 filled 12.3 -> 14.4 us.)
            auto component = [&](int f, WideLifted A, long long B2, long long B3, int EP, int FP, int F2, int F3, int p, int p2, int p3) {
                const int F1 = FP - A.n, FX = max(F2, F3), F = max(F1, FX);
                slow |= (unsigned)(F - max3(F1, p2, p3) + (EP - p) > kWideSlack) << f;
                A.m = wide_shift(A.m, F - F1);
                B2 = wide_shift(B2, F - F2);
                B3 = wide_shift(B3, F - F3);
                long long T;
                if (SCALED) {  // x's sum is the one that is not multiplied
                    T = f == 0 ? A.m + wide_scaled_sum(B2, c.wide_ratio[1], B3, c.wide_ratio[2])
                               : B2 + wide_scaled_sum(A.m, c.wide_ratio[f], B3, c.wide_ratio[3 - f]);
                } else {
                    T = A.m + B2 + B3;
                }
                finish(f, T, EP + F);
            };
            const int hv = c.wide_shift[1], hw = c.wide_shift[2], FU = EU, FV = EV + hv, FW = EW + hw;
            if (DU) {
                const long long aue = wide_align(ue, tu), aus = wide_align(us, tu), aum = wide_align(um, tu);
                const long long q = av0 + ave, qs = avs + wide_align(ves, tv);
                const long long r = aw0 + awe, rb = awm + wide_align(wem, tw);
                component(0, wide_along(aue, auw, au0), wide_across(aun, aus, au0, q, qs),
                          wide_across(aup, aum, au0, r, rb), EU, FU, FV, FW, pu, max3(vx, ve.e, ves.e) + hv, max3(wx, we.e, wem.e) + hw);
            }
            if (DV) {
                const long long avn = wide_align(vn, tv), avw = wide_align(vw, tv), avm = wide_align(vm, tv);
                const long long q = au0 + aun, qw = auw + wide_align(uwn, tu);
                const long long r = aw0 + awn, rb = awm + wide_align(wnm, tw);
                component(1, wide_along(avn, avs, av0), wide_across(ave, avw, av0, q, qw),
                          wide_across(avp, avm, av0, r, rb), EV, FV, FU, FW, pv, max3(ux, un.e, uwn.e), max3(wx, wn.e, wnm.e) + hw);
            }
            if (DW) {
                const long long awp = wide_align(wp, tw), aww = wide_align(ww, tw), aws = wide_align(ws, tw);
                const long long q = au0 + aup, qw = auw + wide_align(uwp, tu);
                const long long r = av0 + avp, rs = avs + wide_align(vsp, tv);
                component(2, wide_along(awp, awm, aw0), wide_across(awe, aww, aw0, q, qw),
                          wide_across(awn, aws, aw0, r, rs), EW, FW, FU, FV, pw, max3(ux, up.e, uwp.e), max3(vx, vp.e, vsp.e) + hv);
            }
            if (DU || DV) {
                wem = we;
                wnm = wn;
            }
            if (NS > 0) {
                // the six faces' velocities at their own largest exponent, in units of the directions' coefficients over x's
                const int E = max3(max(u0.e, uw.e), max(v0.e, vs.e) + hv, max(w0.e, wm.e) + hw);
                const int tu = E + 1, tv = E + (SCALED ? 0 : 1) - hv, tw = E + (SCALED ? 0 : 1) - hw;  // (scaled: halved)
                auto scaled = [&](long long m, int n) { return SCALED ? wide_scale(m, c.wide_ratio[n]) : m; };
                const long long east = wide_shift(u0.m, tu - u0.e), west = -wide_shift(uw.m, tu - uw.e);
                const long long north = wide_shift(scaled(v0.m, 1), tv - v0.e), south = -wide_shift(scaled(vs.m, 1), tv - vs.e);
                const long long top = wide_shift(scaled(w0.m, 2), tw - w0.e), bottom = -wide_shift(scaled(wm.m, 2), tw - wm.e);
#pragma unroll
                for (int n = 0; n < NS; ++n) {
                    const Wide s0 = at(3 + n, 0, 0), se = at(3 + n, 0, 1), sw = at(3 + n, 0, -1), sn = at(3 + n, 1, 0),
                               ss = at(3 + n, -1, 0), sp = over(3 + n, 0, 0), sm = under(3 + n);
                    const int ES = max3(max3(s0.e, se.e, sw.e), max3(sn.e, ss.e, sp.e), sm.e), ts = ES + 2;
                    const long long as0 = wide_align(s0, ts);
                    WideSum sum;
                    sum.add(east, wide_align(se, ts) + as0);
                    sum.add(west, wide_align(sw, ts) + as0);
                    sum.add(north, wide_align(sn, ts) + as0);
                    sum.add(south, wide_align(ss, ts) + as0);
                    sum.add(top, wide_align(sp, ts) + as0);
                    sum.add(bottom, wide_align(sm, ts) + as0);
                    finish(3 + n, sum.value(), ES + E);
                }
            }
            if (max3(EU, EV, EW) >= c.wide_limit) slow = ~0u;
            if (slow) fast_point_fp64<filled, ADVANCE>(a, i, j, k, slow);
        }
        below = slot;
        slot = above;
    }
}

// The tile in the instance's output mode and spacing, both template arguments
// of the loop over the levels: an advance asks for the old values ahead of their
// use and ends in a multiply-add (a filled advance is an advance), and spacings
// whose ratios are no powers of two multiply the directions' sums (a branch at
// each of them instead cost 10 % with either spacing). The plain spacings' loop
// comes first: from behind the other one, its instructions cost a launch on cold
// caches 3 to 20 % (128 x 96 x 40 with a scalar 31.2 us instead of 26.0).
template <int NS, int MASK, int TY>
__device__ __forceinline__ void fast_tile(const AdvArgs &a, int tile_x, int tile_y, int k0, int k1,
                                          long long *smem) {
    auto tile = [&](auto advance) {
        if (!a.f.wide_scaled) fast_tile_mode<NS, MASK, TY, decltype(advance)::value, false>(a, tile_x, tile_y, k0, k1, smem);
        else fast_tile_mode<NS, MASK, TY, decltype(advance)::value, true>(a, tile_x, tile_y, k0, k1, smem);
    };
    if constexpr ((MASK & kFillMask) != 0) {
        tile(std::true_type{});
    } else if (a.mode != 0) {
        tile(std::true_type{});
    } else {
        tile(std::false_type{});
    }
}

#ifdef __CUDACC__
template <int NS, int MASK, int TY, int CTAS = fast_ctas_per_sm<TY>()>
__global__ void __launch_bounds__(fast_threads<TY>(), CTAS)
    advection_fast_kernel(const __grid_constant__ AdvArgs a) {
    extern __shared__ long long wide_smem[];
    const int k0 = blockIdx.z * a.kz;
    fast_tile<NS, MASK, TY>(a, blockIdx.x, blockIdx.y, k0, min(k0 + a.kz, a.nz), wide_smem);
}
#endif

// z-chunk depth of one launch: the one that takes the fewest level-times, waves
// of CTAs times the levels of a chunk and its start (two levels unpacked before
// the first is computed, about a level and a half of time); of equal ones the
// deepest. 256 x 256 x 64: 14 levels, 121 us (8 levels, as four CTAs per SM would
// have, 131); 150 x 100 x 50: 7 levels, 29 us (4: 31, 8: 33).
inline int fast_chunk_depth(int nx, int ny, int nz, int ty, int sms) {
    const long long tiles = (long long)((nx + kFastTX - 1) / kFastTX) * ((ny + ty - 1) / ty);
    const long long slots = (long long)(sms > 0 ? sms : 152) * fast_ctas_per_sm<kFastTY>();
    long long best = -1;
    int depth = 1;
    for (int kz = 1; kz <= kFastKZ && kz <= nz; ++kz) {
        const long long waves = (tiles * ((nz + kz - 1) / kz) + slots - 1) / slots;
        const long long cost = waves * (2 * kz + kFastPrologue);
        if (best < 0 || cost <= best) {
            best = cost;
            depth = kz;
        }
    }
    return depth;
}

#ifdef __CUDACC__
template <int NS, int MASK, int TY>
cudaError_t launch_fast(const AdvArgs &a, int sms, cudaStream_t stream) {
    using Sm = FastSmem<NS, TY>;
    AdvArgs b = a;
    if (b.kz <= 0) b.kz = fast_chunk_depth(b.nx, b.ny, b.nz, TY, sms);
    static std::atomic<unsigned long long> configured{0};
    const auto kernel = advection_fast_kernel<NS, MASK, TY>;
    const cudaError_t e = configure_shared_once(configured, (const void *)kernel, Sm::bytes);
    if (e != cudaSuccess) return e;
    const dim3 block(kFastTX, TY, 1);
    const dim3 grid((b.nx + kFastTX - 1) / kFastTX, (b.ny + TY - 1) / TY, (b.nz + b.kz - 1) / b.kz);
    kernel<<<grid, block, Sm::bytes, stream>>>(b);
    return cudaGetLastError();
}
#endif

} // namespace f2c
