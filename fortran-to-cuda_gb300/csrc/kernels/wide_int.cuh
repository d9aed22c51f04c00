// Stencil arithmetic in 64-bit fixed point at the stencil's own scale.
//
// GB300 issues FP64 at 1.68 lane operations per clock per SM; a 64-bit addition
// is one integer instruction and a 32 x 32 + 64 multiplication another, 64 lanes
// each. A sum of products over neighbouring values therefore costs less in
// integers, provided that they share a scale: FP64 values are unpacked to a
// signed significand and an exponent (Wide), the values of one field that a
// point reads are shifted to the largest exponent among them (wide_align), added
// as integers, and multiplied to the leading 64 bits of the products' sum
// (WideSum), which one conversion and one FP64 product bring back (wide_result).
// No rounding depends on the order of the terms, or on which tile has the point.
//
// Ranges. An unpacked |m| is below 2^63, aligned with a headroom of h bits below
// 2^(63-h). A component's values and the velocities across have h = 3: two
// values' sum or difference is below 2^61, the sums of four below 2^62, f1 + f0 +
// 4c below 6 x 2^60, and a difference is lifted to below 2^62; a direction's
// products add up below 2^61 in the high words and in the middle ones (the low
// word's upper 29 bits), the three directions below 2^62.6. A scalar's values
// have h = 2, its velocities 1: six products of 2^60, middle words of 2^60.
// Dropped: the value bits beyond the alignment's 60 (61), three bits of each low
// word, the low words' product, and the directions' bits below the largest one's
// lowest, together at most 27 and about one unit of 2^-56 times (power of two
// above the largest component value) times (that of the largest velocity across
// or of the difference along).
#pragma once
#include <cuda_runtime.h>

namespace f2c {

constexpr int kWideSpecial = 8192;  // the exponent of infinities and NaN

struct Wide {
    long long m;  // signed significand: 53 bits from bit 62 down
    int e;        // biased exponent
};

// A negative significand one's complemented (2^-62 of it off), zero and
// subnormals without the leading bit, infinities and NaN as kWideSpecial.
__device__ __forceinline__ Wide wide_pack(double x) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const int e = (int)((hi >> 20) & 0x7ffu);
    const long long s = (long long)((int)hi >> 31);
    Wide r;
    r.e = e;
    r.m = (long long)((((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 10) ^ s;
    if ((unsigned)(e - 1) >= 2046u) {
        if (e == 0) {
            r.e = 1;
            r.m = (long long)((((unsigned long long)(hi & 0xfffffu) << 32) | lo) << 10) ^ s;
        } else {
            r.e = kWideSpecial;
        }
    }
    return r;
}

#ifdef __CUDA_ARCH__
// m >> n for any n >= 0 (the PTX shift stops at the width).
__device__ __forceinline__ long long wide_shift(long long m, int n) {
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
    return r;
}
// The words of a significand as 32-bit integers: the high one, and the low one's
// upper 29 bits. Inline PTX, so that the compiler sees plain 32-bit operands and
// multiplies them by the one-instruction 32 x 32 + 64 form; from shifts it knows
// the ranges of, it builds 64 x 64 products instead.
__device__ __forceinline__ int wide_high(long long m) {
    int r;
    asm("{.reg .b32 t; mov.b64 {t, %0}, %1;}" : "=r"(r) : "l"(m));
    return r;
}
__device__ __forceinline__ int wide_low(long long m) {
    int r;
    asm("{.reg .b32 t, u; mov.b64 {t, u}, %1; shr.u32 %0, t, 3;}" : "=r"(r) : "l"(m));
    return r;
}

// m + m as one 64-bit addition (the compiler's own choice, a shift, is two instructions).
__device__ __forceinline__ long long wide_twice(long long m) {
    long long r;
    asm("add.s64 %0, %1, %1;" : "=l"(r) : "l"(m));
    return r;
}
// The left shift that brings the leading bit of d that is not a sign, below bit
// 61, to bit 61; above every exponent where there is none (a zero has no scale).
// A search in each word: the 64-bit one cost registers, which the step spilled
// (512 x 512 x 128 with three scalars 1.75 ms instead of 1.53).
__device__ __forceinline__ int wide_lift(long long d) {
    const int h = wide_high(d);
    unsigned up, low;
    asm("bfind.shiftamt.s32 %0, %1;" : "=r"(up) : "r"(h));
    asm("{.reg .b32 t, u; mov.b64 {t, u}, %1; xor.b32 t, t, u; bfind.shiftamt.u32 %0, t;}" : "=r"(low) : "l"(d));
    return up == ~0u ? (int)(low & 0x1fffu) + 30 : (int)up - 2;
}
// m << n for any n >= 0.
__device__ __forceinline__ long long wide_shift_left(long long m, int n) {
    long long r;
    asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(n));
    return r;
}
// T rounded to 53 bits.
__device__ __forceinline__ double wide_convert(long long T) {
    double t;
    asm("cvt.rn.f64.s64 %0, %1;" : "=d"(t) : "l"(T));
    return t;
}
#else
__device__ __forceinline__ long long wide_shift(long long m, int n) { return m >> (n < 63 ? n : 63); }
__device__ __forceinline__ int wide_high(long long m) { return (int)(m >> 32); }
__device__ __forceinline__ int wide_low(long long m) { return (int)((unsigned)m >> 3); }
__device__ __forceinline__ long long wide_twice(long long m) { return m + m; }
__device__ __forceinline__ int wide_lift(long long d) { const long long m = d < 0 ? ~d : d; return m ? __clzll(m) - 2 : 0x1fff + 30; }
__device__ __forceinline__ long long wide_shift_left(long long m, int n) { return n < 64 ? (long long)((unsigned long long)m << n) : 0; }
__device__ __forceinline__ double wide_convert(long long T) { return (double)T; }
#endif

// The significand at the exponent top - headroom: top is the largest exponent of the stencil plus the headroom.
__device__ __forceinline__ long long wide_align(Wide a, int top) { return wide_shift(a.m, top - a.e); }

__device__ __forceinline__ int max3(int a, int b, int c) { return __vimax3_s32(a, b, c); }

// A sum of products' leading 64 bits.
struct WideSum {
    long long high = 0, middle = 0;
    __device__ __forceinline__ void add(long long a, long long b) {
        const int ah = wide_high(a), bh = wide_high(b);
        const int al = wide_low(a), bl = wide_low(b);
        high += (long long)ah * bh;
        middle += (long long)ah * bl;
        middle += (long long)al * bh;
    }
    __device__ __forceinline__ long long value() const { return high + (middle >> 29); }
};

// A product times 2^(n + 1).
struct WideLifted {
    long long m;
    int n;
};

// A momentum component along its own axis, half its products' sum, with the
// component one cell either side and at the point:
//   (f1 - f0)(f1 + f0 + 4c),
// the difference lifted by n + 1 bits, its leading one to bit 61: in a nearly
// uniform flow it is what is small.
__device__ __forceinline__ WideLifted wide_along(long long f1, long long f0, long long c) {
    WideSum s;
    const long long d = f1 - f0;
    const int lift = wide_lift(d);
    s.add(wide_shift_left(d, lift), (f1 + f0) + wide_twice(wide_twice(c)));
    return {s.value(), lift - 1};
}

// A momentum component across another axis: a1, a0 and c one cell either side of
// the point and there, q, qn the crossing velocity's face sums on the two sides:
//   2(a1 - a0)(q + qn) + (a1 + a0 + 2c)(q - qn).
__device__ __forceinline__ long long wide_across(long long a1, long long a0, long long c, long long q, long long qn) {
    WideSum s;
    s.add(wide_twice(a1 - a0), q + qn);
    s.add((a1 + a0) + wide_twice(c), q - qn);
    return s.value();
}

// m times a significand r in [1/2, 1) (given as 2^63 r), halved.
__device__ __forceinline__ long long wide_scale(long long m, long long r) {
    WideSum s;
    s.add(m, r);
    return s.value();
}
// a times r plus b times t, for |a|, |b| below 2^62 (doubled, for the bits that a product drops).
__device__ __forceinline__ long long wide_scaled_sum(long long a, long long r, long long b, long long t) {
    WideSum s;
    s.add(wide_twice(a), r);
    s.add(wide_twice(b), t);
    return s.value();
}

// T * 2^e * k (plus `old` where ADD), for the coefficient k whose words are
// `khi`, `klo` with the sum's constant 2^-offset taken off the exponent field;
// `ke` is that field less one. The conversion rounds T to 53 bits, the product
// (or multiply-add) rounds once more. Where the factor is below the normal range
// the product is taken 2^512 larger first (the results there are subnormal or
// zero); above it `fits` is cleared, whatever T is: the exponent of an infinity
// or NaN lands there with an ordinary significand, and a T of zero (a flow at
// rest, faces that cancel) says nothing about its product with one.
template <bool ADD>
__device__ __forceinline__ double wide_result(long long T, int e, int khi, int klo, int ke, double old, bool &fits) {
    double t = wide_convert(T);
    fits = true;
    double factor = __hiloint2double(khi + (e << 20), klo);
    if ((unsigned)(e + ke) >= 2046u) {
        if (e + ke >= 2046) fits = false;
        if (e + ke < -500 || T == 0) {
            factor = 0.0;
        } else {
            t *= __hiloint2double(khi + ((e + 512) << 20), klo);
            factor = 0x1p-512;
        }
    }
    return ADD ? __fma_rn(t, factor, old) : t * factor;
}

} // namespace f2c
