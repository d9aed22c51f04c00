// The integer-pipe operations of soft_fp64.cuh by number, for the host's and the device's check
// (tests/test_soft_operations.py); `left` where a range operation leaves its operands to the caller.
#pragma once
#include "soft_fp64.cuh"

namespace soft_cases {
__device__ __forceinline__ double operation(int op, double a, double b, bool &left) {
    left = false;
    if (op == 0) {
        f2c::ProductRange<false> range;
        const double r = f2c::mul_rn_range(a, b, range);
        left = range.left();
        return r;
    }
    if (op == 1) {
        f2c::ProductRange<true> range;
        const double r = f2c::mul_rn_range(a, b, range);
        left = range.left();
        return r;
    }
    if (op == 2) {
        f2c::SumRange range;
        const double r = f2c::add_rn_range(a, b, range);
        left = range.left();
        return r;
    }
    return op == 3 ? f2c::mul_rn_again(a, b) : f2c::add_rn_left(a, b);
}
}  // namespace soft_cases
