// Device check of pivot_inv (csrc/canon.cuh) against the IEEE reciprocal over its declared range
// [1, 2^40]: every exponent with the significands next to all ones and to one (the all-ones
// significand is the one Markstein's correction misses), every integer a pivot of small
// spacings starts from, and pseudo-random significands.  Prints the mismatches (0).
#include <cstdio>
#include <cuda_runtime.h>

#include "../ceemdan-gpu_b200/csrc/canon.cuh"

__device__ void one(double x, unsigned long long* bad) {
    if (__double_as_longlong(ceemdan::pivot_inv(x)) != __double_as_longlong(1.0 / x))
        atomicAdd(bad, 1ull);
}

__global__ void check(unsigned long long* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned long long frac = 0xfffffffffffffull;
    if (t < 4096)
        for (int e = 0; e < 40; ++e) {
            const unsigned long long ex = (unsigned long long)(1023 + e) << 52;
            one(__longlong_as_double((long long)(ex | (frac - t))), bad);
            one(__longlong_as_double((long long)(ex | t)), bad);
        }
    one((double)(t + 1), bad);
    unsigned long long s = 88172645463325252ull + t;
    for (int i = 0; i < 512; ++i) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        const unsigned long long ex = (unsigned long long)(1023 + (int)(s >> 58) % 40) << 52;
        one(__longlong_as_double((long long)(ex | ((s ^ (s >> 31)) & frac))), bad);
    }
}

int main() {
    unsigned long long *bad, h = 1;
    if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(*bad));
    check<<<2048, 256>>>(bad);
    if (cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("mismatches %llu\n", h);
    return h == 0 ? 0 : 1;
}
