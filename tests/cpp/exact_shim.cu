// Device check of csrc/hs_exact.cuh for tests/test_gpu_exact.py: seeded
// operands of one kind, each function against the plain FP64 operation, bit
// for bit.  Returns the number of mismatches, negative on a CUDA error.
#include <cstdint>
#include <cuda_runtime.h>

#include "hs_exact.cuh"

using namespace hsg;
typedef unsigned long long u64;

__device__ u64 next(u64& s) {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    return s * 0x2545F4914F6CDD1Dull;
}
__device__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}

// kinds: 0 any bits, 1 exponents within +-40, 2 short or all-ones mantissas,
// 3 quotients next to 1, 4 quotients next to a midpoint of two doubles
__global__ void check(int kind, u64 seed, int n, u64* bad) {
    u64 s = seed * 0x9E3779B97F4A7C15ull + (blockIdx.x * (u64)blockDim.x + threadIdx.x) * 0xD1342543DE82EF95ull + 1;
    for (int i = 0; i < 4; ++i) next(s);
    const u64 mant = 0x000FFFFFFFFFFFFFull, one = 0x3FF0000000000000ull;
    u64 miss = 0;
    for (int i = 0; i < n; ++i) {
        u64 a = next(s), b = next(s);
        if (kind == 1) {
            a = (a & ~0x7FF0000000000000ull) | ((983 + next(s) % 81) << 52);
            b = (b & ~0x7FF0000000000000ull) | ((983 + next(s) % 81) << 52);
        } else if (kind >= 2) {
            a = (a & mant) | one;
            b = (b & mant) | one;
            if (kind == 2) {
                if (next(s) & 1) a &= ~0ull << (next(s) % 53);
                if (next(s) & 1) b &= ~0ull << (next(s) % 53);
                if ((next(s) & 3) == 0) b |= (1ull << (next(s) % 52)) - 1;
            } else if (kind == 3) {
                a = b + (long long)(next(s) % 4097) - 2048;
                if (next(s) & 1) a = b + (long long)(next(s) >> (18 + next(s) % 20)) - (1ll << 25);
            } else {
                a = __double_as_longlong(__longlong_as_double(a) * __longlong_as_double(b)) + (long long)(next(s) % 5) - 2;
            }
        }
        const double x = __longlong_as_double(a), d = __longlong_as_double(b);
        miss += !same(quotient(x, d), x / d);
        miss += lessThan(x, d) != (x < d) || atMost(x, d) != (x <= d) || atMost(x, x) != (x <= x);
        miss += isZero(x) != (x == 0.0) || isOne(x) != (x == 1.0);
        if (kind == 1 || kind == 2) {
            const double y = __drcp_rn(d);
            miss += !same(quotientBy(x, d, y), x / d);
            const double v = fabs(x) * 1000.0;
            if (v < 2147483648.0) {
                double f;
                const uint32_t k = splitFraction(v, f);
                miss += k != (uint32_t)v || !same(f, v - (uint32_t)v);
            }
        }
    }
    if (miss) atomicAdd(bad, miss);
}

extern "C" long long exact_check(int kind, u64 seed, int blocks, int n) {
    u64 *d = nullptr, h = 0;
    if (cudaMalloc(&d, 8) != cudaSuccess || cudaMemset(d, 0, 8) != cudaSuccess) return -1;
    check<<<blocks, 256>>>(kind, seed, n, d);
    if (cudaDeviceSynchronize() != cudaSuccess) return -2;
    cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (long long)h;
}
