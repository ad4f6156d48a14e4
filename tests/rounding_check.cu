// Compares the packed reciprocal, square root and division of the libm mode
// (csrc/bsg_math.cuh) with the correctly rounded functions, bit for bit, over
// the ranges that the mode uses them in (compiled by tests/test_rounding.py).
// Each call returns the number of differences and leaves one of them in *bad.
#include "bsg_math.cuh"

namespace {

__device__ unsigned long long g_count;
__device__ unsigned long long g_bad;

__device__ __forceinline__ void compare(float got, float want, uint32_t a, uint32_t b) {
    if (__float_as_uint(got) == __float_as_uint(want)) return;
    atomicAdd(&g_count, 1ull);
    g_bad = (unsigned long long)a << 32 | b;
}

// Every float from lo (its bits) on, `count` of them, two neighbours at a time.
template <bool SQRT>
__global__ void unary_kernel(uint32_t lo, uint32_t count) {
    const uint64_t step = 2ull * gridDim.x * blockDim.x;
    for (uint64_t i = 2ull * (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x); i + 1 < count; i += step) {
        const uint32_t u0 = lo + (uint32_t)i, u1 = u0 + 1;
        const float2 x = make_float2(__uint_as_float(u0), __uint_as_float(u1));
        const float2 y = SQRT ? bsg::sqrt2_rn(x) : bsg::rcp2_rn(x);
        compare(y.x, SQRT ? __fsqrt_rn(x.x) : __frcp_rn(x.x), u0, 0);
        compare(y.y, SQRT ? __fsqrt_rn(x.y) : __frcp_rn(x.y), u1, 0);
    }
}

__device__ __forceinline__ uint64_t mix(uint64_t x) {  // splitmix64's output function
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// A dividend and a divisor of exponents in [-30, 30] and [-45, 45].
// kind 0: random significands; 1: both within 32 units of a power of two;
// 2: a quotient next to the middle of two floats.
__device__ __forceinline__ float2 pair_of(uint64_t h, int kind) {
    uint32_t ma = (uint32_t)h & 0x7FFFFFu, mb = (uint32_t)(h >> 23) & 0x7FFFFFu;
    const uint32_t ea = 127 - 30 + (uint32_t)(h >> 46) % 61, eb = 127 - 45 + (uint32_t)(h >> 54) % 91;
    if (kind == 1) {
        ma = ((ma & 63) - 32) & 0x7FFFFFu;
        mb = ((mb & 63) - 32) & 0x7FFFFFu;
    }
    const float b = __uint_as_float(eb << 23 | mb);
    float a = __uint_as_float(ea << 23 | ma);
    if (kind == 2) {  // a = b (q + half a unit), as near as a float is
        const double q = (double)__uint_as_float(127u << 23 | ma) + 5.9604644775390625e-8;
        const double p = (double)__uint_as_float(127u << 23 | mb) * q;
        a = __uint_as_float(ea << 23) * (float)p;
    }
    return make_float2(a, b);
}

__global__ void div_kernel(uint64_t first, uint64_t count, int kind) {
    const uint64_t step = 2ull * gridDim.x * blockDim.x;
    for (uint64_t i = 2ull * (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x); i + 1 < count; i += step) {
        const float2 x = pair_of(mix(first + i), kind), y = pair_of(mix(first + i + 1), kind);
        const float2 q = bsg::div2_rn(make_float2(x.x, y.x), make_float2(x.y, y.y));
        compare(q.x, __fdiv_rn(x.x, x.y), __float_as_uint(x.x), __float_as_uint(x.y));
        compare(q.y, __fdiv_rn(y.x, y.y), __float_as_uint(y.x), __float_as_uint(y.y));
    }
}

constexpr int kGrid = 1216, kBlock = 256;

long long result(unsigned long long* bad) {
    unsigned long long n = 0;
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(&n, g_count, 8) != cudaSuccess ||
        cudaMemcpyFromSymbol(bad, g_bad, 8) != cudaSuccess)
        return -1;
    return (long long)n;
}

bool reset() {
    const unsigned long long zero = 0;
    return cudaMemcpyToSymbol(g_count, &zero, 8) == cudaSuccess && cudaMemcpyToSymbol(g_bad, &zero, 8) == cudaSuccess;
}

}  // namespace

// Every float in [2^from, 2^to).
extern "C" long long check_unary(int sqrt, int from, int to, unsigned long long* bad) {
    if (from < -126 || to > 128 || from >= to || !reset()) return -1;
    for (int e = from; e < to; ++e) {
        const uint32_t lo = (uint32_t)(e + 127) << 23;
        if (sqrt) unary_kernel<true><<<kGrid, kBlock>>>(lo, 1u << 23);
        else unary_kernel<false><<<kGrid, kBlock>>>(lo, 1u << 23);
    }
    return result(bad);
}

// launches x 2^30 pairs of a kind (pair_of).
extern "C" long long check_div(unsigned long long seed, int launches, int kind, unsigned long long* bad) {
    if (kind < 0 || kind > 2 || !reset()) return -1;
    for (int j = 0; j < launches; ++j)
        div_kernel<<<kGrid, kBlock>>>((seed << 40) + ((uint64_t)j << 30), 1ull << 30, kind);
    return result(bad);
}
