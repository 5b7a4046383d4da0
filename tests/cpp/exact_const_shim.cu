// Device check of csrc/hs_exact.cuh's division by a constant for
// tests/test_gpu_exact_const.py: dividends next to q d and to the midpoint
// between q and the next double times d, for any q and for q with all ones or
// few bits, against the plain division, bit for bit.  Returns the number of
// mismatches, negative on a CUDA error.
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

__global__ void check(double dGiven, u64 seed, int n, u64* bad) {
    u64 s = seed * 0x9E3779B97F4A7C15ull + (blockIdx.x * (u64)blockDim.x + threadIdx.x) * 0xD1342543DE82EF95ull + 1;
    for (int i = 0; i < 4; ++i) next(s);
    u64 miss = 0;
    for (int i = 0; i < n; ++i) {
        u64 q = (next(s) & 0x000FFFFFFFFFFFFFull) | ((1013 + next(s) % 21) << 52);
        if ((next(s) & 3) == 0) q |= (1ull << (next(s) % 52)) - 1;
        if ((next(s) & 3) == 0) q &= ~0ull << (next(s) % 53);
        double d = dGiven;
        if (d == 0.0) {             // any divisor, its mantissa all ones or short at times
            u64 b = (next(s) & 0x000FFFFFFFFFFFFFull) | ((1003 + next(s) % 41) << 52);
            if ((next(s) & 3) == 0) b |= (1ull << (next(s) % 52)) - 1;
            if ((next(s) & 3) == 0) b &= ~0ull << (next(s) % 53);
            d = __longlong_as_double((long long)b);
        }
        const double y = 1.0 / d, Q = __longlong_as_double((long long)q);
        const double half = __longlong_as_double((long long)((q & 0x7FF0000000000000ull) - (53ull << 52)));
        // the product, or the product with the midpoint above q, rounded; then places beside it
        double a = (next(s) & 1) ? __fma_rn(half, d, Q * d) : Q * d;
        a = __longlong_as_double(__double_as_longlong(a) + (long long)(next(s) % 7) - 3);
        const double got = quotientBy(a, d, y), want = a / d;
        miss += __double_as_longlong(got) != __double_as_longlong(want);
    }
    if (miss) atomicAdd(bad, miss);
}

extern "C" long long exact_const_check(double d, u64 seed, int blocks, int n) {
    u64 *p = nullptr, h = 0;
    if (cudaMalloc(&p, 8) != cudaSuccess || cudaMemset(p, 0, 8) != cudaSuccess) return -1;
    check<<<blocks, 256>>>(d, seed, n, p);
    if (cudaDeviceSynchronize() != cudaSuccess) return -2;
    cudaMemcpy(&h, p, 8, cudaMemcpyDeviceToHost);
    cudaFree(p);
    return (long long)h;
}
