// Device check of the divisions of the sift kernels (csrc/spline_device.cuh) against the IEEE
// division, bit for bit (any NaN for a NaN): rcp_raw and div_int for integer divisors h and 3h,
// seg_coeffs_int for segments of h samples.  h: every length up to 4096, and pseudo-random ones up to
// 2^31 (3h up to 2^33); dividends: pseudo-random over the whole range of exponents, multiples of the
// divisor and their neighbours, zeros, subnormals, the largest numbers, infinities and NaN.
// Prints the mismatches (0) of each.
#include <cstdio>
#include <cuda_runtime.h>

#include "../ceemdan-gpu_b200/csrc/spline_device.cuh"

namespace {
struct Rng {
    unsigned long long s;
    __device__ unsigned long long next() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return s ^ (s >> 29);
    }
};
__device__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}
__device__ double from_bits(unsigned long long b) { return __longlong_as_double((long long)b); }

// dividend k of divisor d
__device__ double dividend(Rng& r, int k, double d) {
    const unsigned long long u = r.next(), sign = u & 0x8000000000000000ull;
    const unsigned long long frac = r.next() >> 12;
    switch (k & 7) {
        case 0: return from_bits(sign | (u >> 3 & 0x7ff) << 52 | frac);  // any exponent
        case 1: {  // next to a multiple of d
            const double m = d * (double)(long long)(u >> 20 & 0xfffffff) * 0x1p-11;
            return from_bits((unsigned long long)__double_as_longlong(m) + (u & 3) - 1);
        }
        case 2: {
            const double sp[8] = {0.0, -0.0, 0x1p-1074, -0x1.8p-1030, 0x1.fffffffffffffp+1023,
                                  -INFINITY, NAN, 0x1p-960};
            return sp[u >> 7 & 7];
        }
        case 3: return from_bits(sign | (u >> 3 & 0x3f) << 52 | frac);           // tiny
        case 4: return from_bits(sign | (0x7c0 + (u >> 3 & 0x3f)) << 52 | frac);  // huge
        default: return from_bits(sign | (1023 - 40 + (u >> 3) % 80) << 52 | frac);
    }
}
}  // namespace

__global__ void check(unsigned long long* bad) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    Rng r{88172645463325252ull + 7919ull * t};
    for (int i = 0; i < 64; ++i) {
        const double h = t < 4096 ? (double)(t + 1) : (double)(1 + (r.next() >> 33));
        for (int three = 0; three < 2; ++three) {
            const double d = three ? 3.0 * h : h;
            if (!same(ceemdan::rcp_raw(d), 1.0 / d)) atomicAdd(&bad[0], 1ull);
            const double a = dividend(r, i, d);
            if (!same(ceemdan::div_int(a, d), a / d)) atomicAdd(&bad[1], 1ull);
        }
        const double slope = dividend(r, i + 1, h), c0 = dividend(r, i + 2, h),
                     c1 = dividend(r, i + 2, h);
        double b, d;
        ceemdan::seg_coeffs_int(h, slope, c0, c1, b, d);
        if (!same(b, slope - (h * fma(2.0, c0, c1)) / 3.0) || !same(d, (c1 - c0) / (3.0 * h)))
            atomicAdd(&bad[2], 1ull);
    }
}

int main() {
    unsigned long long *bad, h[3] = {1, 1, 1};
    if (cudaMalloc(&bad, sizeof(h)) != cudaSuccess) return 2;
    cudaMemset(bad, 0, sizeof(h));
    check<<<1024, 256>>>(bad);
    if (cudaMemcpy(h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    std::printf("mismatches %llu %llu %llu\n", h[0], h[1], h[2]);
    return h[0] + h[1] + h[2] == 0 ? 0 : 1;
}
