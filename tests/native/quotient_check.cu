// Compares the quotients of gral_b200/csrc/prog_quot.cuh with plain divisions on the device, bit for bit
// (NaN equal to NaN).  One line per check, its name and the number of mismatches; "divided" counts operands
// of a physical range that needed the division, of which there must be none.
#include <cstdint>
#include <cstdio>

#include "prog_quot.cuh"

using namespace gral;

namespace {

typedef unsigned long long u64;

__device__ u64 mix(u64 z) {       // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ bool same(float a, float b) { return (a != a && b != b) || __float_as_uint(a) == __float_as_uint(b); }
__device__ bool same(double a, double b) {
    return (a != a && b != b) || __double_as_longlong(a) == __double_as_longlong(b);
}
__device__ void count(u64 *c, bool bad) {
    if (bad) atomicAdd(c, 1ull);
}
// a float with an exponent field in [lo, hi], every sixteenth with a significand next to a power of two
__device__ float pick(u64 r, int lo, int hi) {
    unsigned m = (unsigned)r & 0x7fffff;
    if ((r >> 24 & 15) == 0) m = (r >> 28 & 1) ? (m & 3) : 0x7fffff - (m & 3);
    const unsigned e = (unsigned)(lo + (int)((r >> 32 & 0xffff) % (unsigned)(hi - lo + 1)));
    return __uint_as_float(((unsigned)(r >> 63) << 31) | (e << 23) | m);
}
__device__ double pickd(u64 r, u64 r2, int lo, int hi) {
    u64 m = r & 0xfffffffffffffull;
    if ((r2 >> 24 & 15) == 0) m = (r2 >> 28 & 1) ? (m & 3) : 0xfffffffffffffull - (m & 3);
    const u64 e = (u64)(lo + (int)((r2 >> 32 & 0xffff) % (unsigned)(hi - lo + 1)));
    return __longlong_as_double((long long)((r2 >> 63 << 63) | (e << 52) | m));
}
__device__ float guarded(float x, float d, bool &divided) {
    float q = 0.0f;
    quot_if(q, x, d, 1.0f / d, 1u);
    divided = odd_divisor(d) || odd_quotient(x, q);
    return divided ? x / d : q;
}
__device__ double guarded(double x, double d, bool &divided) {
    double q = 0.0;
    quot_if(q, x, d, 1.0 / d, 1u);
    divided = odd_divisor(d) || odd_quotient(x, q);
    return divided ? x / d : q;
}

// every divisor from 2^-27 to 2^43
__global__ void k_rcp(u64 *c) {
    for (u64 b = 0x32000000u + (u64)blockIdx.x * blockDim.x + threadIdx.x; b < 0x55000000u; b += (u64)gridDim.x * blockDim.x) {
        const float d = __uint_as_float((unsigned)b);
        count(c, !same(rcp_rn(d), 1.0f / d));
    }
}
__global__ void k_random(u64 *c, u64 n) {
    for (u64 t = (u64)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (u64)gridDim.x * blockDim.x) {
        const u64 r = mix(4 * t), s = mix(4 * t + 1), r2 = mix(4 * t + 2), s2 = mix(4 * t + 3);
        bool div;
        {   // dividend 2^-60 .. 2^60, divisor 2^-27 .. 2^35: inside the range
            const float x = pick(r, 67, 187), d = fabsf(pick(s, 100, 162));
            count(c, !same(quot(x, d, rcp_rn(d)), x / d));
            count(c + 1, !same(guarded(x, d, div), x / d));
            count(c + 2, div);
            const double xd = pickd(r, r2, 1023 - 500, 1023 + 500), dd = fabs(pickd(s, s2, 1023 - 127, 1023 + 127));
            count(c + 3, !same(guarded(xd, dd, div), xd / dd));
            count(c + 4, div);
        }
        {   // any dividend, any divisor
            const float x = pick(r, 0, 255), d = pick(s, 0, 255);
            count(c + 5, !same(guarded(x, d, div), x / d));
            const double xd = pickd(r, r2, 0, 2047), dd = pickd(s, s2, 0, 2047);
            count(c + 6, !same(guarded(xd, dd, div), xd / dd));
            // div_by: positive divisors with a normal reciprocal
            const float p = fabsf(pick(s, 2, 252));
            count(c + 7, !same(div_by(x, p, 1.0f / p), x / p));
        }
        {   // around the ends of the dividend's and the quotient's range
            const float d = fabsf(pick(s, 60, 194));
            const bool low = r >> 40 & 1, quotient = r >> 41 & 1;
            int e = low ? 27 : 224;
            if (quotient) e += (int)(__float_as_uint(d) >> 23) - 127;
            e += (int)(r >> 42 & 7) - 4;
            const float x = __uint_as_float((unsigned)min(max(e, 0), 255) << 23 | ((unsigned)r & 0x7fffff));
            count(c + 5, !same(guarded(x, d, div), x / d));
            count(c + 7, !same(div_by(x, d, 1.0f / d), x / d));
        }
    }
}
// every pair of special values
__constant__ float F[20] = {0.0f, -0.0f, 1.0f, -1.0f, 3.0f, 1e-45f, -1e-45f, 1.17549421e-38f, 1.17549435e-38f, 7.8886091e-31f,
                            7.8886086e-31f, 1.58456325e29f, 3.40282347e38f, -3.40282347e38f, 8.6736174e-19f, 1.15292150e18f,
                            1.15292160e18f, 1e-4f, 8000.0f, 0.3f};
__global__ void k_special(u64 *c) {
    const float inf = __uint_as_float(0x7f800000u), nan = __uint_as_float(0x7fc00000u);
    auto val = [&](int q) { return q < 20 ? F[q] : (q == 20 ? inf : (q == 21 ? -inf : nan)); };
    if (threadIdx.x >= 23) return;
    bool div;
    for (int q = 0; q < 23; ++q) {
        const float x = val(threadIdx.x), d = val(q);
        count(c, !same(guarded(x, d, div), x / d));
        count(c + 1, !same(guarded((double)x, (double)d, div), (double)x / (double)d));
        if (d > 1e-37f && d < 1e37f) count(c + 2, !same(div_by(x, d, 1.0f / d), x / d));
    }
}

}  // namespace

int main() {
    u64 *c = nullptr, h[12] = {0};
    const u64 n = 1ull << 28;
    if (cudaMalloc((void **)&c, sizeof(h)) != cudaSuccess || cudaMemset(c, 0, sizeof(h)) != cudaSuccess) return 2;
    k_rcp<<<1480, 256>>>(c);
    k_random<<<1480, 256>>>(c + 1, n);
    k_special<<<1, 32>>>(c + 9);
    if (cudaMemcpy(h, c, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    const char *names[12] = {"rcp_rn",       "quot",     "quot_if",       "divided",         "quot_if_double", "divided_double",
                             "quot_if_any",  "quot_if_double_any", "div_by", "special", "special_double",  "special_div_by"};
    for (int q = 0; q < 12; ++q) std::printf("%s %llu\n", names[q], h[q]);
    cudaFree(c);
    return 0;
}
