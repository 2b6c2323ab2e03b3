// The float square root and quotient of the subgrid rate in the 16-bit kernels
// (sqrt_normal, two_over_normal: a hardware estimate and one correction)
// against the correctly rounded functions, for every float of their ranges;
// and dev_rate, which chooses between them and the general functions, against
// the general expression for arguments of every kind.
// Exit status 1 and the counts on a mismatch, 2 on a CUDA error.
#include <cstdio>

#include "lbm_kernels.cuh"

using namespace lbm;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }

// bad: mismatches of the root, the quotient, the rate.
__global__ void check(unsigned long long *bad) {
    const unsigned long long at = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x,
                             step = (unsigned long long)gridDim.x * blockDim.x;
    unsigned long long n[3] = {0, 0, 0};
    for (unsigned long long i = 0x0D800000u + at; i < 0x71800000u; i += step) {  // [2^-100, 2^100)
        const float x = __uint_as_float((unsigned)i);
        n[0] += !same(sqrt_normal(x), sqrtf(x));
    }
    for (unsigned long long i = 0x3E800000u + at; i < 0x5D800000u; i += step) {  // [2^-2, 2^60)
        const float x = __uint_as_float((unsigned)i);
        n[1] += !same(two_over_normal(x), 2.0f / x);
    }
    // q: a share of all bit patterns (zero, subnormals, negatives, infinities and not-a-numbers among them)
    const float tau[6] = {0.5f, 0.51f, 0.953575f, 3.0f, 0x1p40f, 0x1p62f}, c[5] = {0.0f, 0.735f, 25.0f, -0.5f, 0x1p90f};
    for (unsigned long long i = at * 16; i < (1ull << 32); i += step * 16) {
        const float q = __uint_as_float((unsigned)i + (unsigned)(i >> 9 & 15));
        for (int t = 0; t < 6; t++)
            for (int k = 0; k < 5; k++) {
                const float want = 2.0f / (tau[t] + sqrtf(__fmaf_rn(c[k], sqrtf(q), __fmul_rn(tau[t], tau[t]))));
                n[2] += !same(dev_rate<float>(q, tau[t], c[k]), want);
            }
    }
    for (int k = 0; k < 3; k++)
        if (n[k]) atomicAdd(&bad[k], n[k]);
}

int main() {
    unsigned long long *d = nullptr, h[3] = {1, 1, 1};
    if (cudaMalloc(&d, sizeof(h)) || cudaMemset(d, 0, sizeof(h))) return 2;
    check<<<2048, 256>>>(d);
    if (cudaGetLastError() || cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost)) return 2;
    cudaFree(d);
    printf("mismatches: square root %llu, quotient %llu, rate %llu\n", h[0], h[1], h[2]);
    return h[0] || h[1] || h[2];
}
