// Generality stencils on the same z-march / 2-D tile machinery as the
// advection templates, FP64 with the reference grouping (bit-identical to the
// oracle):
//   diffusion7: compiler/tests/apps/box/stepper.f90:8-30
//       b = a + dt*nu*((a(i-1)+a(i+1)+a(j-1)+a(j+1)+a(k-1)+a(k+1) - 6*a)/(dx*dx))
//   jacobi5:    compiler/tests/apps/relax/relax.f90:28-33
//       v = 0.25*(u(i-1)+u(i+1)+u(j-1)+u(j+1))
//   yee2d:      2-D TM leapfrog (this project's form; no reference source in the mount)
//       Hx -= ch*(Ez(j+1)-Ez); Hy += ch*(Ez(i+1)-Ez); then Ez += ce*((Hy-Hy(i-1)) - (Hx-Hx(j-1)))
// Dirichlet-zero boundaries are ghost values kept at zero; no kernel writes a ghost.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "soft_fp64.cuh"

// FP64 additions bound these stencils (1.68 lanes a clock per SM), so the
// products and as many additions as balance the two run on the integer pipes
// (soft_fp64.cuh; the correctly rounded results, the same bits), without
// branches: a point whose operands they cannot take is done again in FP64. The
// additions moved are ones along y: a zero of the west or east boundary would
// send a warp of every row that way, one of the others only the outer rows'.
namespace f2c {

// x * 2^e for an exact power-of-two factor, on the integer pipe when the
// result stays normal (the same bits as the correctly rounded product);
// the FP64 multiply otherwise.
// The multiplication for the rare operands the exponent shift cannot take. Out
// of line, so that the common path issues no FP64 instruction (an inline
// fallback is evaluated alongside and costs one FP64 multiply per point).
static __device__ __noinline__ double scale_by(double x, double factor) { return x * factor; }

__device__ __forceinline__ double scale_pow2(double x, int e, double factor) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)((unsigned long long)b >> 52) & 0x7ff;
    const int r = ex + e;
    if (ex != 0 && ex != 0x7ff && r >= 1 && r <= 0x7fe) return __longlong_as_double(b + ((long long)e << 52));
    return scale_by(x, factor);
}

// IEEE negation on the integer pipe (a plain -x here becomes an FP64 addition).
__device__ __forceinline__ double sign_flipped(double x) {
    unsigned long long r;
    asm("xor.b64 %0, %1, 0x8000000000000000;" : "=l"(r) : "l"((unsigned long long)__double_as_longlong(x)));
    return __longlong_as_double((long long)r);
}

// The division where dx*dx is no power of two, out of line (inline it is evaluated for every point).
static __device__ __noinline__ double divide(double x, double y) { return x / y; }

struct DiffusionArgs {
    const double *a;
    double *b;
    double dtnu;      // dt*nu, formed on the host exactly as the source does
    double dx2;       // dx*dx
    int dx2_pow2;     // dx*dx is 2^dx2_exp: the division is an exact scaling
    int dx2_exp;
    int nx, ny, nz, h;
    long long sx, plane;
};

constexpr int kDiffBX = 32, kDiffBY = 8, kDiffKZ = 32;

// 384^3: 0.59 ms with two of the seven additions on the integer pipes (0.79 with
// none, 0.70 with one, 0.69 with three: an addition there takes 50 ALU
// instructions, an FP64 one the time of 38).
static __global__ void __launch_bounds__(kDiffBX *kDiffBY) diffusion7_kernel(const DiffusionArgs p) {
    const int i = blockIdx.x * kDiffBX + threadIdx.x;
    const int j = blockIdx.y * kDiffBY + threadIdx.y;
    if (i >= p.nx || j >= p.ny) return;
    const int k0 = blockIdx.z * kDiffKZ;
    const int k1 = min(k0 + kDiffKZ, p.nz);
    const double *__restrict__ A = p.a;
    const long long sx = p.sx, plane = p.plane;
    long long q = (long long)(i + p.h) + sx * (long long)(j + p.h) + plane * (long long)(k0 + p.h);
    double below = __ldg(A + q - plane), centre = __ldg(A + q);
    // an exact scaling commutes with the product after it (its operand within 2^-511 .. 2^511, the scale within 2^-256 .. 2^256)
    const bool folded = p.dx2_pow2 && p.dx2_exp >= -256 && p.dx2_exp <= 256;
    const double factor = folded ? scale_pow2(p.dtnu, -p.dx2_exp, 1.0 / p.dx2) : p.dtnu;
    for (int k = k0; k < k1; ++k, q += plane) {
        const double west = __ldg(A + q - 1), east = __ldg(A + q + 1), south = __ldg(A + q - sx), north = __ldg(A + q + sx);
        const double above = __ldg(A + q + plane);
        ProductRange<false> range;
        SumRange sums;
        const double first = add_rn_range(add_rn_range(west + east, south, sums), north, sums);
        const double num = (first + below + above) - mul_rn_range(6.0, centre, range);
        const double lap = folded ? num : divide(num, p.dx2);
        double r = centre + mul_rn_range(factor, lap, range);
        if (range.left() || sums.left()) {
            const double n = add_rn_hw(add_rn_hw(add_rn_hw(west, east), south), north) + below + above - mul_rn_hw(6.0, centre);
            r = centre + mul_rn_hw(p.dtnu, p.dx2_pow2 ? scale_pow2(n, -p.dx2_exp, 1.0 / p.dx2) : n / p.dx2);
        }
        p.b[q] = r;
        below = centre;
        centre = above;
    }
}

struct JacobiArgs {
    const double *u;
    double *v;
    int nx, ny, h;
    long long sx;
};

constexpr int kJacBX = 64, kJacBY = 4, kJacJY = 8;  // each thread does kJacJY rows

// 8192^2: 0.27 ms with one of the three additions on the integer pipes (0.39 with
// none, 0.34 with three in two rows).
static __global__ void __launch_bounds__(kJacBX *kJacBY) jacobi5_kernel(const JacobiArgs p) {
    const int i = blockIdx.x * kJacBX + threadIdx.x;
    const int j0 = (blockIdx.y * kJacBY + threadIdx.y) * kJacJY;
    if (i >= p.nx) return;
    const double *__restrict__ U = p.u;
    const long long sx = p.sx;
    long long q = (long long)(i + p.h) + sx * (long long)(j0 + p.h);
    const int j1 = min(j0 + kJacJY, p.ny);
    double south = j0 < p.ny ? __ldg(U + q - sx) : 0.0;
    double centre = j0 < p.ny ? __ldg(U + q) : 0.0;
    for (int j = j0; j < j1; ++j, q += sx) {
        const double north = __ldg(U + q + sx), west = __ldg(U + q - 1), east = __ldg(U + q + 1);
        SumRange sums;
        const double across = west + east;
        double three = add_rn_range(across, south, sums);
        if (sums.left()) three = add_rn_hw(across, south);
        p.v[q] = scale_pow2(three + north, -2, 0.25);
        south = centre;
        centre = north;
    }
}

struct YeeArgs {
    double *ez, *hx, *hy;
    double ch, ce;
    int nx, ny, h;
    long long sx;
};

// 4096^2: 0.245 ms a step with one addition of four on the integer pipes in each kernel (0.14 + 0.11; 0.28 with none).
constexpr int kYeeBX = 64, kYeeBY = 4, kYeeJY = 2;  // each thread does kYeeJY rows

static __global__ void __launch_bounds__(kYeeBX *kYeeBY) yee_h_kernel(const YeeArgs p) {
    const int i = blockIdx.x * kYeeBX + threadIdx.x;
    const int j0 = (blockIdx.y * kYeeBY + threadIdx.y) * kYeeJY;
    if (i >= p.nx || j0 >= p.ny) return;
    long long q = (long long)(i + p.h) + p.sx * (long long)(j0 + p.h);
    const int j1 = min(j0 + kYeeJY, p.ny);
    double e = __ldg(p.ez + q);
#pragma unroll
    for (int j = j0; j < j0 + kYeeJY; ++j, q += p.sx) {
        if (j >= j1) return;
        const double north = __ldg(p.ez + q + p.sx), east = __ldg(p.ez + q + 1);
        const double hx = p.hx[q], hy = p.hy[q];
        ProductRange<false> range;
        SumRange sums;
        double x = hx - mul_rn_range(p.ch, add_rn_range(north, sign_flipped(e), sums), range);
        double y = hy + mul_rn_range(p.ch, east - e, range);
        if (range.left() || sums.left()) {
            x = hx - mul_rn_hw(p.ch, north - e);
            y = hy + mul_rn_hw(p.ch, east - e);
        }
        p.hx[q] = x;
        p.hy[q] = y;
        e = north;
    }
}

static __global__ void __launch_bounds__(kYeeBX *kYeeBY) yee_e_kernel(const YeeArgs p) {
    const int i = blockIdx.x * kYeeBX + threadIdx.x;
    const int j0 = (blockIdx.y * kYeeBY + threadIdx.y) * kYeeJY;
    if (i >= p.nx || j0 >= p.ny) return;
    long long q = (long long)(i + p.h) + p.sx * (long long)(j0 + p.h);
    const int j1 = min(j0 + kYeeJY, p.ny);
    double south = __ldg(p.hx + q - p.sx);
#pragma unroll
    for (int j = j0; j < j0 + kYeeJY; ++j, q += p.sx) {
        if (j >= j1) return;
        const double ez = p.ez[q], hy = __ldg(p.hy + q), west = __ldg(p.hy + q - 1), hx = __ldg(p.hx + q);
        ProductRange<false> range;
        SumRange sums;
        double e = ez + mul_rn_range(p.ce, (hy - west) - add_rn_range(hx, sign_flipped(south), sums), range);
        if (range.left() || sums.left()) e = ez + mul_rn_hw(p.ce, (hy - west) - (hx - south));
        p.ez[q] = e;
        south = hx;
    }
}

inline dim3 diffusion_grid(const DiffusionArgs &p) {
    return dim3((p.nx + kDiffBX - 1) / kDiffBX, (p.ny + kDiffBY - 1) / kDiffBY, (p.nz + kDiffKZ - 1) / kDiffKZ);
}
inline dim3 jacobi_grid(const JacobiArgs &p) {
    return dim3((p.nx + kJacBX - 1) / kJacBX, (p.ny + kJacBY * kJacJY - 1) / (kJacBY * kJacJY), 1);
}
inline dim3 yee_grid(const YeeArgs &p) { return dim3((p.nx + kYeeBX - 1) / kYeeBX, (p.ny + kYeeBY * kYeeJY - 1) / (kYeeBY * kYeeJY), 1); }

// Exponent e with x == 2^e exactly, or a flag that x is not a power of two.
inline bool power_of_two(double x, int *e) {
    if (!(x > 0.0)) return false;
    int k = 0;
    double m = x;
    while (m >= 2.0 && k < 1100) { m *= 0.5; ++k; }
    while (m < 1.0 && k > -1100) { m *= 2.0; --k; }
    if (m != 1.0) return false;
    *e = k;
    return true;
}

} // namespace f2c
