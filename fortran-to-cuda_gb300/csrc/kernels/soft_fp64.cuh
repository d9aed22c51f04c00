// Binary64 addition and multiplication on the integer pipes, rounded to
// nearest-even exactly as IEEE 754-2019 (clauses 4.3.1 and 5.4.1) defines them.
//
// GB300 issues FP64 at 1.68 lane operations per clock per SM, while its integer
// pipes take 64 (shifts, logic, compares and 64-bit additions on the ALU pipe,
// wide multiplications on the FMA pipe), at the same time: some 38 ALU
// instructions run in the time of one FP64 operation. The kernels bound by FP64
// move products (22 ALU instructions) and some additions (50) there. The
// results are the correctly rounded ones, so they equal the hardware's DADD and
// DMUL bit for bit: substituting one for the other changes no value.
//
// The method is the textbook one (align, add or subtract the significands with
// a sticky bit jammed into the lowest position, normalise, round to nearest with
// ties to even; the product's significand as a 106-bit integer), written without
// branches for the common operands: a branch in each operation keeps the
// compiler from interleaving independent ones. Operands that it does not take
// (zeros, subnormals, infinities, NaN, the ends of the exponent range; all rare
// in the stencils' fields) are noted, and the caller does the point again in
// FP64. Doubles are taken apart as 32-bit words throughout: masking the sign of
// a double's 64-bit pattern is compiled into an FP64 |x|, two FP64 instructions
// in an addition meant to save one.
#pragma once
#include <cuda_runtime.h>

namespace f2c {

// The cases the integer paths leave out, kept out of line: a call stays a
// branch that only lanes needing it take, where an inline hardware operation
// would be if-converted into an FP64 instruction that every lane issues.
static __device__ __noinline__ double add_rn_hw(double a, double b) { return __dadd_rn(a, b); }
static __device__ __noinline__ double mul_rn_hw(double a, double b) { return __dmul_rn(a, b); }

// Words of a 64-bit pattern. On the device they are inline PTX: where the
// compiler sees a word as a shift of a value whose range it knows, it multiplies
// 64 x 64 bits instead of 32 x 32.
#ifdef __CUDA_ARCH__
__device__ __forceinline__ unsigned high_word(unsigned long long x) {
    unsigned r;
    asm("{.reg .b32 t; mov.b64 {t, %0}, %1;}" : "=r"(r) : "l"(x));
    return r;
}
__device__ __forceinline__ unsigned low_word(unsigned long long x) {
    unsigned r;
    asm("{.reg .b32 t; mov.b64 {%0, t}, %1;}" : "=r"(r) : "l"(x));
    return r;
}
// (h:l + inc * 2^-32) with `top` added to the high word: inc is a carry-in's 32-bit addend below the low word.
__device__ __forceinline__ unsigned long long add_carry(unsigned h, unsigned l, unsigned below, unsigned inc, unsigned top) {
    unsigned long long r;
    asm("{.reg .b32 t, u, v; add.cc.u32 t, %3, %4; addc.cc.u32 u, %2, 0; addc.u32 v, %1, %5; mov.b64 %0, {u, v};}"
        : "=l"(r) : "r"(h), "r"(l), "r"(below), "r"(inc), "r"(top));
    return r;
}
#else
inline unsigned high_word(unsigned long long x) { return (unsigned)(x >> 32); }
inline unsigned low_word(unsigned long long x) { return (unsigned)x; }
inline unsigned long long add_carry(unsigned h, unsigned l, unsigned below, unsigned inc, unsigned top) {
    return (((unsigned long long)h << 32) | l) + (((unsigned long long)below + inc) >> 32) + ((unsigned long long)top << 32);
}
#endif
// The high word of hi:lo << n, for n in 1..31.
__device__ __forceinline__ unsigned shl_high(unsigned hi, unsigned lo, unsigned n) { return (hi << n) | (lo >> (32u - n)); }

// What the products below collect over any number of them: operands within
// 2^-511 .. 2^511 are taken, whose product is normal; WIDE takes every normal
// operand of a product well inside the normal range (two instructions more).
template <bool WIDE>
struct ProductRange {
    unsigned operand = 0, result = 0;  // largest distance (as unsigned numbers) from the lowest exponent taken
    __device__ __forceinline__ bool left() const {
        return operand >= (WIDE ? 0x7FE00000u : 0x3FF00000u) || result >= 0x7FC00000u;
    }
};

// a * b, rounded to nearest-even, without a branch; `range` tells the caller,
// after any number of products, that an operand was not taken, and that they are
// to be done again in FP64.
template <bool WIDE>
__device__ __forceinline__ double mul_rn_range(double a, double b, ProductRange<WIDE> &range) {
    const unsigned long long ia = (unsigned long long)__double_as_longlong(a);
    const unsigned long long ib = (unsigned long long)__double_as_longlong(b);
    const unsigned ahi = high_word(ia), alo = low_word(ia), bhi = high_word(ib), blo = low_word(ib);
    const unsigned ea = ahi & 0x7FF00000u, eb = bhi & 0x7FF00000u;  // the exponent fields, in place
    const unsigned least = WIDE ? 0x00100000u : 0x20000000u;
    const unsigned ra = ea - least, rb = eb - least, r2 = ra > rb ? ra : rb;
    range.operand = range.operand > r2 ? range.operand : r2;
    if (WIDE) {
        const unsigned re = ea + eb - (1024u << 20);
        range.result = range.result > re ? range.result : re;
    }
    // significands, a's shifted left by 10: the product's high 64 bits h1:h0 lie in [2^50, 2^52), and the
    // middle word's sum stays below 2^64
    const unsigned ah = (shl_high(ahi, alo, 10) & 0x3FFFFFFFu) | 0x40000000u, al = alo << 10;
    const unsigned bh = (bhi & 0xFFFFFu) | 0x100000u, bl = blo;
    const unsigned long long low = (unsigned long long)al * bl;
    const unsigned long long mid = (unsigned long long)ah * bl + (unsigned long long)al * bh + high_word(low);
    const unsigned long long high = (unsigned long long)ah * bh + high_word(mid);
    const unsigned l0 = low_word(low);
    unsigned l1 = low_word(mid) | (l0 < 1u ? l0 : 1u);  // the word below, the lowest one jammed into it
    unsigned h1 = high_word(high), h0 = low_word(high);
    const unsigned z = 2u - (h1 >> 19);  // left shift that brings the leading one to bit 52
    h1 = shl_high(h1, h0, z);
    h0 = shl_high(h0, l1, z);
    l1 <<= z;
    // rounds up when the word below is over half, or half with h0 odd; the leading one adds to the exponent field
    const unsigned long long r = add_carry(h1, h0, l1, 0x7FFFFFFFu + (h0 & 1u), ea + eb - (z << 20) - (1022u << 20));
    return __longlong_as_double((long long)(r | ((unsigned long long)((ahi ^ bhi) & 0x80000000u) << 32)));
}

// What add_rn_range collects over any number of additions.
struct SumRange {
    unsigned apart = 0, end = 0;  // largest exponent difference, and distance below 2^-959 (unsigned)
    int top = 63;                 // lowest leading bit of a sum (-1: zero)
    __device__ __forceinline__ bool left() const { return apart > 0x01F00000u || end > 0x77000000u || top < 0; }
};

// a + b, rounded to nearest-even, without a branch, for operands between 2^-959
// and 2^945 at most 2^31 apart, with a sum that is not zero; `range` collects
// what tells the caller that one was not so, and that the sums are to be done
// again in FP64.
__device__ __forceinline__ double add_rn_range(double a, double b, SumRange &range) {
    const unsigned long long ia = (unsigned long long)__double_as_longlong(a);
    const unsigned long long ib = (unsigned long long)__double_as_longlong(b);
    const unsigned ahi = high_word(ia), alo = low_word(ia), bhi = high_word(ib), blo = low_word(ib);
    // the larger magnitude first (compared as words: a sign cleared in a double's 64 bits becomes an FP64 |x|)
    const unsigned ha = ahi & 0x7FFFFFFFu, hb = bhi & 0x7FFFFFFFu;
    const bool swap = (((unsigned long long)ha << 32) | alo) < (((unsigned long long)hb << 32) | blo);
    const unsigned xh = swap ? bhi : ahi, xl = swap ? blo : alo, yh = swap ? ahi : bhi, yl = swap ? alo : blo;
    const unsigned xe = xh & 0x7FF00000u, ye = yh & 0x7FF00000u, apart = xe - ye, end = ye - 0x04000000u;
    range.apart = range.apart > apart ? range.apart : apart;
    range.end = range.end > end ? range.end : end;
    // significands with the leading bit at 61; the smaller one, a bit higher, shifted right by one and the
    // exponents' difference as a product by 2^(31 - difference), what that drops jammed into the lowest bit
    const unsigned long long x = ((unsigned long long)((shl_high(xh, xl, 9) & 0x1FFFFFFFu) | 0x20000000u) << 32) | (xl << 9);
    const unsigned sh = (shl_high(yh, yl, 10) & 0x3FFFFFFFu) | 0x40000000u, sl = yl << 10, f = 0x80000000u >> ((apart >> 20) & 31u);
    const unsigned long long low = (unsigned long long)sl * f, high = (unsigned long long)sh * f + high_word(low);
    const unsigned lost = low_word(low), less = (unsigned)((int)(xh ^ yh) >> 31);
    const unsigned long long y = ((unsigned long long)(high_word(high) ^ less) << 32) | ((low_word(high) | (lost < 1u ? lost : 1u)) ^ less);
    const unsigned long long s = x + y - (unsigned long long)(long long)(int)less;
    const int top = 63 - __clzll((long long)s);
    range.top = range.top < top ? range.top : top;
    const unsigned long long n = s << ((62 - top) & 63);
    const unsigned h0 = low_word(n);
    const unsigned long long r = (n + (0x1FFu + ((h0 >> 10) & 1u))) >> 10;
    return __longlong_as_double((long long)(r + ((unsigned long long)((xh & 0xFFF00000u) + ((unsigned)(top - 62) << 20)) << 32)));
}

// A product that mul_rn_range left, done again: of a zero (fields at rest and
// plateaus are made of them) on the integer pipes as well, others in FP64.
__device__ __forceinline__ bool is_zero(double x) {
    const unsigned long long i = (unsigned long long)__double_as_longlong(x);
    return ((high_word(i) << 1) | low_word(i)) == 0;
}
__device__ __forceinline__ bool is_finite(double x) {
    return (high_word((unsigned long long)__double_as_longlong(x)) & 0x7FF00000u) != 0x7FF00000u;
}
__device__ __forceinline__ double mul_rn_left(double a, double b) {
    if ((is_zero(a) && is_finite(b)) || (is_zero(b) && is_finite(a)))
        return __longlong_as_double((__double_as_longlong(a) ^ __double_as_longlong(b)) & (long long)0x8000000000000000ULL);
    return mul_rn_hw(a, b);
}
// A sum that add_rn_range left, done again in the same way: with a zero, and of opposite numbers.
__device__ __forceinline__ double add_rn_left(double a, double b) {
    const long long ia = __double_as_longlong(a), ib = __double_as_longlong(b);
    if (is_finite(a) && is_finite(b)) {
        if (is_zero(a)) return is_zero(b) ? __longlong_as_double(ia & ib) : b;
        if (is_zero(b)) return a;
        if ((ia ^ ib) == (long long)0x8000000000000000ULL) return 0.0;
    }
    return add_rn_hw(a, b);
}
// Out of line, for kernels whose common path would otherwise make room for it.
static __device__ __noinline__ double mul_rn_again(double a, double b) { return mul_rn_left(a, b); }

// One operation by itself, operands outside the range going to the hardware's (the kernels use the forms above, which
// leave that to the end of several).
__device__ __forceinline__ double add_rn_int(double a, double b) {
    SumRange range;
    const double r = add_rn_range(a, b, range);
    return range.left() ? add_rn_hw(a, b) : r;
}
// add_rn_int for operands of nearby exponents, which need no other path.
__device__ __forceinline__ double add_rn_near(double a, double b) { return add_rn_int(a, b); }
__device__ __forceinline__ double mul_rn_int(double a, double b) {
    ProductRange<false> range;
    const double r = mul_rn_range(a, b, range);
    return range.left() ? mul_rn_hw(a, b) : r;
}

} // namespace f2c
