// Host check of the branch-free integer-pipe sum and product (soft_fp64.cuh:
// add_rn_range, mul_rn_range) against the host's IEEE doubles, over the operand
// pairs of cases.h: equal bit for bit wherever they do not leave the operands to
// FP64, and left only outside the ranges they state.
// Usage: soft_fp64_range_host <pairs per distribution>; exit status 1 on a mismatch.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#define __device__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
using std::min;
static inline long long __double_as_longlong(double d) { long long x; std::memcpy(&x, &d, 8); return x; }
static inline double __longlong_as_double(long long x) { double d; std::memcpy(&d, &x, 8); return d; }
static inline double __dadd_rn(double a, double b) { volatile double r = a + b; return r; }
static inline double __dmul_rn(double a, double b) { volatile double r = a * b; return r; }
static inline int __clzll(long long x) { return x == 0 ? 64 : __builtin_clzll((unsigned long long)x); }

#include "soft_fp64.cuh"
#include "cases.h"

int main(int argc, char **argv) {
    const uint64_t n = argc > 1 ? std::strtoull(argv[1], nullptr, 10) : 1000000;
    int failed = 0;
    for (int op = 0; op < 3; ++op)
        for (int dist = 0; dist < 7; ++dist)
            for (uint64_t i = 0; i < n; ++i) {
                uint64_t ia, ib;
                soft_cases::pair(dist, 0x5eed1000ull + 131 * (uint64_t)dist + (uint64_t)op, i, &ia, &ib);
                const double a = __longlong_as_double((long long)ia), b = __longlong_as_double((long long)ib);
                const int ea = (int)(ia >> 52) & 0x7FF, eb = (int)(ib >> 52) & 0x7FF;
                const double want = op ? __dmul_rn(a, b) : __dadd_rn(a, b);
                double got;
                bool left, may;
                if (op == 1) {
                    f2c::ProductRange<false> range;
                    got = f2c::mul_rn_range(a, b, range);
                    left = range.left();
                    may = ea < 512 || ea > 1534 || eb < 512 || eb > 1534;
                } else if (op == 2) {
                    f2c::ProductRange<true> range;
                    got = f2c::mul_rn_range(a, b, range);
                    left = range.left();
                    may = ea == 0 || eb == 0 || ea == 0x7FF || eb == 0x7FF || ea + eb < 1024 || ea + eb >= 1024 + 2044;
                } else {
                    f2c::SumRange range;
                    got = f2c::add_rn_range(a, b, range);
                    left = range.left();
                    may = std::abs(ea - eb) > 31 || std::min(ea, eb) < 64 || std::min(ea, eb) > 1968 || want == 0.0;
                }
                const bool wrong = left ? !may : may || __double_as_longlong(got) != __double_as_longlong(want);
                if (wrong && failed++ < 4) std::printf("op %d dist %d: %a %a -> %a, not %a (left %d)\n", op, dist, a, b, got, want, left);
            }
    return failed != 0;
}
