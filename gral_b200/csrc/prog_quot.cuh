// prog_quot.cuh -- correctly rounded quotients without the compiler's range checks and their branches.
//
// With y = RN(1/d), q1 = q0 + (x - d*q0)*y is within an ulp of x/d and RN(q1 + (x - d*q1)*y) is the IEEE
// quotient (P. Markstein, IBM J. Res. Dev. 34(1), 1990), while no remainder leaves the subnormal range
// and nothing overflows.  For a positive float d that holds while x and the quotient both lie within
// 2^-100 .. 2^97: a remainder is a multiple of ulp(d)*ulp(q) >= 2^-147.  Outside it the
// callers divide.  A quotient costs 5 operations and several may share a divisor.  tests/native/
// quotient_check.cu compares all of this with plain divisions on the device.
#pragma once

#include <cuda_runtime.h>

namespace gral {

// 1/d of a divisor in [2^-27, 2^43): one Newton step on the hardware's approximation, compared with the
// division for every value of that range.
__device__ __forceinline__ float rcp_rn(float d) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
    return fmaf(fmaf(-d, y, 1.0f), y, y);
}
__device__ __forceinline__ float quot(float x, float d, float y) {
    float q = x * y;
    q = fmaf(fmaf(-d, q, x), y, q);
    return fmaf(fmaf(-d, q, x), y, q);
}

// The worse of a dividend's and its computed quotient's place in the range, which is below QUOT_SPAN where
// the quotient is the IEEE quotient; a zero dividend gives zero.  Integer operations only: tested value by
// value, with the branches that brings, a k-eps iteration on 100x90 took 1.15 ms instead of 0.99.  Doubles by
// their upper words, 2^-900 .. 2^892.
constexpr unsigned QUOT_SPAN = 0x62800000u, QUOT_SPAN_DOUBLE = 0x70000000u;
__device__ __forceinline__ unsigned quot_worst(float x, float q) {
    const unsigned w = max((__float_as_uint(x) & 0x7fffffffu) - 0x0d800000u, (__float_as_uint(q) & 0x7fffffffu) - 0x0d800000u);
    return x == 0.0f ? 0u : w;
}
__device__ __forceinline__ unsigned quot_worst(double x, double q) {
    const unsigned w = max((unsigned)(__double2hiint(x) & 0x7fffffff) - 0x07b00000u,
                           (unsigned)(__double2hiint(q) & 0x7fffffff) - 0x07b00000u);
    return x == 0.0 ? 0u : w;
}
// a dividend and its computed quotient that may not be the IEEE quotient
__device__ __forceinline__ bool odd_quotient(float x, float q) { return quot_worst(x, q) >= QUOT_SPAN; }
__device__ __forceinline__ bool odd_quotient(double x, double q) { return quot_worst(x, q) >= QUOT_SPAN_DOUBLE; }
// a divisor whose quotients may not be: outside 2^-60 .. 2^60 (in double 2^-127 .. 2^129) or negative
__device__ __forceinline__ bool odd_divisor(float d) { return __float_as_uint(d) - 0x21800000u >= 0x3c000000u; }
__device__ __forceinline__ bool odd_divisor(double d) { return (unsigned)__double2hiint(d) - 0x38000000u >= 0x10000000u; }

// x/d with y = RN(1/d) for any x and a positive d whose reciprocal is a normal number: the quotient above
// in its range, zero as it is, and the plain division for the rest.
__device__ __forceinline__ float div_by(float x, float d, float y) {
    const float q = quot(x, d, y);
    if (odd_quotient(x, q)) return x / d;
    return x == 0.0f ? x : q;
}

// q = x/d where `on`, with y = RN(1/d); the last operation and the zero case are predicated
__device__ __forceinline__ void quot_if(float &q, float x, float d, float y, unsigned on) {
    float q1 = x * y;
    q1 = fmaf(fmaf(-d, q1, x), y, q1);
    const float r = fmaf(-d, q1, x);
    asm("{\n\t.reg .pred f, n;\n\tsetp.ne.u32 f, %5, 0;\n\tsetp.neu.and.f32 n, %1, 0f00000000, f;\n\t"
        "@f mov.f32 %0, %1;\n\t@n fma.rn.f32 %0, %2, %3, %4;\n\t}"
        : "+f"(q)
        : "f"(x), "f"(r), "f"(y), "f"(q1), "r"(on));
}
__device__ __forceinline__ void quot_if(double &q, double x, double d, double y, unsigned on) {
    double q1 = x * y;
    q1 = fma(fma(-d, q1, x), y, q1);
    const double r = fma(-d, q1, x);
    asm("{\n\t.reg .pred f, n;\n\tsetp.ne.u32 f, %5, 0;\n\tsetp.neu.and.f64 n, %1, 0d0000000000000000, f;\n\t"
        "@f mov.f64 %0, %1;\n\t@n fma.rn.f64 %0, %2, %3, %4;\n\t}"
        : "+d"(q)
        : "d"(x), "d"(r), "d"(y), "d"(q1), "r"(on));
}

}  // namespace gral
