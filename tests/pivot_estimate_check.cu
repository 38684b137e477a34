// The estimate that rcp_raw (csrc/canon.cuh) starts from: the largest |1 - x y0| over every leading
// 20 bits of the significand with the other bits clear and set, at both ends of the pivots' range of
// exponents.  Then pivot_inv against the IEEE reciprocal at the significands whose reciprocals lie
// closest to a midpoint between doubles (see tests/test_reciprocal_rounding.py), at every exponent.
// Prints the largest error in units of 2^-18 as a percentage, and the mismatches (0).
#include <cstdio>
#include <cstdlib>
#include <cuda_runtime.h>

#include "../ceemdan-gpu_b200/csrc/canon.cuh"

__global__ void estimate(unsigned long long* most) {
    const unsigned long long lead = blockIdx.x * blockDim.x + threadIdx.x;
    for (int e = 0; e <= 40; e += 40)
        for (int set = 0; set < 2; ++set) {
            const unsigned long long bits = (unsigned long long)(1023 + e) << 52 | lead << 32 |
                                            (set ? 0xffffffffull : 0ull);
            const double x = __longlong_as_double((long long)bits);
            double y;
            asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
            const double err = fabs(fma(-x, y, 1.0)) * 0x1p+18;
            atomicMax(most, (unsigned long long)ceil(err * 100.0));
        }
}

__global__ void near_midpoints(const unsigned long long* sig, int n, unsigned long long* bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int e = 0; e < 40; ++e) {
        const unsigned long long bits =
            (unsigned long long)(1023 + e) << 52 | (sig[i] & 0xfffffffffffffull);
        const double x = __longlong_as_double((long long)bits);
        if (__double_as_longlong(ceemdan::pivot_inv(x)) != __double_as_longlong(1.0 / x))
            atomicAdd(bad, 1ull);
    }
}

int main(int argc, char** argv) {
    unsigned long long *d = nullptr, h[2] = {0, 1}, sig[64], *ds = nullptr;
    const int n = argc - 1 < 64 ? argc - 1 : 64;
    if (n < 1) return 2;
    for (int i = 0; i < n; ++i) sig[i] = std::strtoull(argv[1 + i], nullptr, 10);
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess || cudaMalloc(&ds, sizeof(sig)) != cudaSuccess)
        return 2;
    cudaMemset(d, 0, sizeof(h));
    cudaMemcpy(ds, sig, sizeof(sig[0]) * n, cudaMemcpyHostToDevice);
    estimate<<<(1 << 20) / 256, 256>>>(d);
    near_midpoints<<<1, 64>>>(ds, n, d + 1);
    if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("percent %llu mismatches %llu\n", h[0], h[1]);
    return h[0] < 100 && h[1] == 0 ? 0 : 1;
}
