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

#include <cmath>
#include <cstdint>

#include "device.cuh"
#include "soft_fp64.cuh"

// FP64 additions bound these stencils (1.68 lanes a clock per SM), so the
// products and as many additions as balance the two run on the integer pipes
// (soft_fp64.cuh; the correctly rounded results, the same bits), without
// branches: a point whose operands they cannot take is done again in FP64. The
// additions moved are ones along y: a zero of the west or east boundary would
// send a warp of every row that way, one of the others only the outer rows'.
// A diffusion warp that sees a zero among the values its integer operations
// would read (a region at rest, an outer row) goes to FP64 at once instead of
// doing the point twice: 256^3 of zeros 0.48 -> 0.33 ms with dx 1, 1.63 -> 0.33
// with dx 0.3. In the Yee kernels the same choice costs fields without zeros more
// (0.238 -> 0.249 ms at 4096^2); there a point done again leaves products of zeros
// to the integers (mul_rn_again). 4096^2 at rest: 0.37-0.38 ms with every sum in
// FP64, 0.40-0.41 with FP64 products in the points done again, 0.32 now; fields of
// plateaus, whose points mix both, 0.31-0.33, 0.40-0.41 and 0.37.
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
    if (((unsigned long long)b << 1) == 0) return x;  // (the factor is 2^e)
    return scale_by(x, factor);
}

// IEEE negation on the integer pipe (a plain -x here becomes an FP64 addition).
__device__ __forceinline__ double sign_flipped(double x) {
    unsigned long long r;
    asm("xor.b64 %0, %1, 0x8000000000000000;" : "=l"(r) : "l"((unsigned long long)__double_as_longlong(x)));
    return __longlong_as_double((long long)r);
}

// A value whose high word is zero but for the sign: zero, or far below what the integer operations take.
__device__ __forceinline__ bool nearly_zero(unsigned a, unsigned b, unsigned c) { return min(min(a << 1, b << 1), c << 1) == 0; }

// The division where dx*dx is no power of two, out of line (inline it is evaluated for every point).
static __device__ __noinline__ double divide(double x, double y) { return x / y; }
// The same where y > 0 (dx*dx and not NaN), without a zero numerator's slow path: 0 / y is that zero.
__device__ __forceinline__ double quotient(double x, double y, bool positive) {
    if (positive && ((unsigned long long)__double_as_longlong(x) << 1) == 0) return x;
    return divide(x, y);
}

// x / b, correctly rounded, for a divisor b known to the host, with `high` the
// rounded reciprocal and `low` what that leaves (reciprocal_of): the quotient to
// half a unit and a little (x low + x high, Brisebarre, Muller and Raina 2004),
// its exact remainder, and Markstein's last step (1990), which rounds correctly
// from any quotient within a unit and a correctly rounded reciprocal. For x within
// 2^-511 .. 2^511 and b within 2^-256 .. 2^256 nothing leaves the normal range.
// Three FP64 operations (its first product is on the integer pipes) instead of a
// division's call: 256^3 with dx 0.3 0.40 -> 0.31 ms.
__device__ __forceinline__ double divide_by(double x, double b, double high, double low, ProductRange<false> &range) {
    const double q = __fma_rn(x, high, mul_rn_range(x, low, range));
    return __fma_rn(__fma_rn(-q, b, x), high, q);
}

struct DiffusionArgs {
    const double *a;
    double *b;
    double dtnu;      // dt*nu, formed on the host exactly as the source does
    double dx2;       // dx*dx
    int dx2_positive; // dx*dx > 0 (a NaN is not)
    int dx2_pow2;     // dx*dx is 2^dx2_exp: the division is an exact scaling
    int dx2_exp;
    double high, low; // 1/(dx*dx) as two doubles where it divides by them (else zeros)
    int nx, ny, nz, h;
    long long sx, plane;
    int kz;           // levels per z-chunk (diffusion_grid)
};

constexpr int kDiffBX = 32, kDiffBY = 8, kDiffKZ = 32;

// The point in FP64 (one call, so that the common path issues none of it).
static __device__ __noinline__ double diffusion_fp64(const DiffusionArgs &p, double west, double east, double south, double north,
                                                     double below, double above, double centre) {
    const double n = west + east + south + north + below + above - 6.0 * centre;
    const long long b = __double_as_longlong(n);
    const int ex = (int)((unsigned long long)b >> 52) & 0x7ff, r = ex - p.dx2_exp;
    double lap;
    if (p.dx2_pow2 && ex != 0 && ex != 0x7ff && r >= 1 && r <= 0x7fe) lap = __longlong_as_double(b - ((long long)p.dx2_exp << 52));
    else lap = quotient(n, p.dx2, p.dx2_positive);
    return centre + p.dtnu * lap;
}

// 384^3: 0.575 ms (0.59 before the chunk depths and the choice above) with two of the seven additions on the integer pipes (0.79 with
// none, 0.70 with one, 0.69 with three: an addition there takes 50 ALU
// instructions, an FP64 one the time of 38). A plateau's points, whose zero
// quotient the last product does not take, need no more than their value: 256^3
// constant 0.18 ms (0.31-0.32 with none, 0.46-0.48 done again).
static __global__ void __launch_bounds__(kDiffBX *kDiffBY) diffusion7_kernel(const __grid_constant__ DiffusionArgs p) {
    const int i = blockIdx.x * kDiffBX + threadIdx.x;
    const int j = blockIdx.y * kDiffBY + threadIdx.y;
    const bool active = i < p.nx && j < p.ny;
    const unsigned lanes = __ballot_sync(0xffffffffu, active);
    if (!active) return;
    const int k0 = blockIdx.z * p.kz;
    const int k1 = min(k0 + p.kz, p.nz);
    const double *__restrict__ A = p.a;
    const long long sx = p.sx, plane = p.plane;
    long long q = (long long)(i + p.h) + sx * (long long)(j + p.h) + plane * (long long)(k0 + p.h);
    double below = __ldg(A + q - plane), centre = __ldg(A + q);
    // an exact scaling commutes with the product after it (its operand within 2^-511 .. 2^511, the scale within 2^-256 .. 2^256)
    const bool folded = p.dx2_pow2 && p.dx2_exp >= -256 && p.dx2_exp <= 256;
    const double factor = folded ? scale_pow2(p.dtnu, -p.dx2_exp, 1.0 / p.dx2) : p.dtnu;
    const bool known = p.high != 0.0;
    const bool exact = (folded || known) && is_finite(p.dtnu);  // whose dt*nu times zero over dx^2 is zero
    for (int k = k0; k < k1; ++k, q += plane) {
        const double west = __ldg(A + q - 1), east = __ldg(A + q + 1), south = __ldg(A + q - sx), north = __ldg(A + q + sx);
        const double above = __ldg(A + q + plane);
        bool again = __any_sync(lanes, nearly_zero((unsigned)__double2hiint(centre), (unsigned)__double2hiint(south),
                                                   (unsigned)__double2hiint(north)));
        double r;
        bool flat = false;  // a plateau: the sums cancel, and the value stays as it is
        if (!again) {
            ProductRange<false> range;
            SumRange sums;
            const double first = add_rn_range(add_rn_range(west + east, south, sums), north, sums);
            const double num = (first + below + above) - mul_rn_range(6.0, centre, range);
            const double lap = folded ? num : (known ? divide_by(num, p.dx2, p.high, p.low, range) : divide(num, p.dx2));
            r = centre + mul_rn_range(factor, lap, range);
            again = range.left() || sums.left();
            flat = exact && !sums.left() && is_zero(num);
        }
        if (again) {
            // (e: the centre's 6.0 * centre was taken)
            const unsigned e = (unsigned)__double2hiint(centre) & 0x7FF00000u;
            if (flat && e - 0x20000000u < 0x3FF00000u) r = centre;
            else r = diffusion_fp64(p, west, east, south, north, below, above, centre);
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
    int rows;  // rows a thread does (jacobi_grid)
};

constexpr int kJacBX = 64, kJacBY = 4, kJacJY = 8;  // most rows a thread does

// 8192^2: 0.27 ms with one of the three additions on the integer pipes (0.39 with
// none, 0.34 with three in two rows). At rest 0.39 (0.54 with every sum in FP64
// or with a zero's sums and scaling done again there).
static __global__ void __launch_bounds__(kJacBX *kJacBY) jacobi5_kernel(const JacobiArgs p) {
    const int i = blockIdx.x * kJacBX + threadIdx.x;
    const int j0 = (blockIdx.y * kJacBY + threadIdx.y) * p.rows;
    if (i >= p.nx) return;
    const double *__restrict__ U = p.u;
    const long long sx = p.sx;
    long long q = (long long)(i + p.h) + sx * (long long)(j0 + p.h);
    const int j1 = min(j0 + p.rows, p.ny);
    double south = j0 < p.ny ? __ldg(U + q - sx) : 0.0;
    double centre = j0 < p.ny ? __ldg(U + q) : 0.0;
    for (int j = j0; j < j1; ++j, q += sx) {
        const double north = __ldg(U + q + sx), west = __ldg(U + q - 1), east = __ldg(U + q + 1);
        SumRange sums;
        const double across = west + east;
        double three = add_rn_range(across, south, sums);
        if (sums.left()) three = add_rn_left(across, south);
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
            x = hx - mul_rn_again(p.ch, north - e);
            y = hy + mul_rn_again(p.ch, east - e);
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
        if (range.left() || sums.left()) e = ez + mul_rn_again(p.ce, (hy - west) - (hx - south));
        p.ez[q] = e;
        south = hx;
    }
}

// Levels of a z-chunk: the depth with the least time on the SM with the most
// CTAs, as the strict advection kernel's (chunk_depth); a deep march on a small
// grid is one long serial chain. 26 x 26 x 156: 7.8 us a step (23 at 32 levels, with
// every addition in FP64).
inline dim3 diffusion_grid(DiffusionArgs &p) {
    const unsigned gx = (p.nx + kDiffBX - 1) / kDiffBX, gy = (p.ny + kDiffBY - 1) / kDiffBY;
    const long long sms = current_sm_count();
    long long best = -1;
    for (int kz = 1; kz <= kDiffKZ && kz <= p.nz; ++kz) {
        const long long ctas = (long long)gx * gy * ((p.nz + kz - 1) / kz);
        const long long cost = ((ctas + sms - 1) / sms + 1) * (2 * kz + 1);
        if (best < 0 || cost <= best) {
            best = cost;
            p.kz = kz;
        }
    }
    return dim3(gx, gy, (p.nz + p.kz - 1) / p.kz);
}
// Rows of a thread: as many (8, 4, 2 or 1) as leave kJacCtas CTAs per SM; the
// rows of a thread are one serial chain. 251 x 5541: 10.4 us a sweep (13.1 at 8 rows,
// with every addition in FP64).
constexpr int kJacCtas = 8;
inline dim3 jacobi_grid(JacobiArgs &p) {
    const unsigned gx = (p.nx + kJacBX - 1) / kJacBX;
    const long long wanted = (long long)kJacCtas * current_sm_count();
    p.rows = kJacJY;
    while (p.rows > 1 && (long long)gx * ((p.ny + kJacBY * p.rows - 1) / (kJacBY * p.rows)) < wanted) p.rows /= 2;
    return dim3(gx, (p.ny + kJacBY * p.rows - 1) / (kJacBY * p.rows), 1);
}
inline dim3 yee_grid(const YeeArgs &p) { return dim3((p.nx + kYeeBX - 1) / kYeeBX, (p.ny + kYeeBY * kYeeJY - 1) / (kYeeBY * kYeeJY), 1); }

// The reciprocal of b as two doubles, rounded and its remainder, for divide_by;
// false where b is not one that it takes (a power of two among them: no remainder).
inline bool reciprocal_of(double b, double *high, double *low) {
    *high = *low = 0.0;
    if (!(b >= 0x1p-256 && b <= 0x1p256)) return false;
    const double h = 1.0 / b, l = std::fma(-h, b, 1.0) / b;
    if (!(std::fabs(l) >= 0x1p-500)) return false;
    *high = h;
    *low = l;
    return true;
}

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
