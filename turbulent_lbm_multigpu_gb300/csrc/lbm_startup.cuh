// lbm_startup.cuh -- the seeded start-up velocity and a cavity's first state.
#pragma once
#include "lbm_kernels.cuh"

namespace lbm {

// Philox4x32-10 (Salmon et al., SC'11), same as the oracle's.
__device__ __forceinline__ void philox(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c[0];
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * c[2];
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c[1] ^ k0;
        const uint32_t n1 = (uint32_t)p1;
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c[3] ^ k1;
        const uint32_t n3 = (uint32_t)p0;
        c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
}

// (2 unit - 1) as a double, unit = (r >> 8) 2^-24: an even integer of 25 bits
// over 2^24, so a float holds it and widening is bit placement.  The FP64
// pipe (1.75 lanes per clock and SM, conversions included) is left with one
// product per component of the 18 operations that the plain expression takes.
__device__ __forceinline__ double signed_unit(uint32_t r) {
    const float f = (float)((int32_t)((r >> 8) << 1) - 16777216) * 0x1p-24f;
    const uint32_t b = __float_as_uint(f), m = b & 0x7fffffffu;
    return m ? double_of(((m >> 3) + 0x38000000u) | (b & 0x80000000u), b << 29) : 0.0;
}
// A double to float, to nearest even; magnitudes of normal floats by bits.
template <typename R> __device__ __forceinline__ R to_real(double v);
template <> __device__ __forceinline__ double to_real<double>(double v) { return v; }
template <> __device__ __forceinline__ float to_real<float>(double v) {
    const uint64_t b = bits_of(v);
    const uint32_t hi = hi32(b) & 0x7fffffffu, lo = (uint32_t)b;
    if (hi - 0x38100000u >= 0x47C00000u - 0x38100000u) return (float)v;  // outside [2^-126, 2^125): zero too
    const uint64_t s = join(hi, lo) + 0x0fffffffu + ((lo >> 29) & 1u);
    return __uint_as_float(shl2((uint32_t)s, hi32(s) - 0x38000000u, 3) | (hi32(b) & 0x80000000u));
}

// Start-up velocity of a physical cell, uniform on [-amp, amp) per component.
template <typename R> __device__ __forceinline__ void startup_velocity(uint64_t idx, uint64_t seed, double amp, R u[3]) {
    uint32_t r[4] = {(uint32_t)idx, (uint32_t)(idx >> 32), 0u, 0u};
    philox(r, (uint32_t)seed, (uint32_t)(seed >> 32));
#pragma unroll
    for (int a = 0; a < 3; a++) u[a] = to_real<R>(signed_unit(r[a]) * amp);
}

// A lid-driven cavity at step 0 in one pass: walls on all faces (which win
// over the lid plane, CController::setGeometry, src/CController.hpp:531-546),
// the seeded start-up in the slot order that the first (beta) step reads.
// As init, the lid's flags and the start-up one after the other would leave
// it, at one store per population instead of two.
template <typename S>
__global__ void __launch_bounds__(256) k_cavity(LatDesc d, uint64_t seed, double amp, int store_v) {
    using R = typename Store<S>::R;
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= d.n) return;
    const uint32_t cc = (uint32_t)c, nx = (uint32_t)d.nx, ny = (uint32_t)d.ny, nz = (uint32_t)d.nz;
    const uint32_t row = cc / nx, x = cc - row * nx, z = row / ny, y = row - z * ny;
    const bool inside = x > 0 && y > 0 && z > 0 && x < nx - 1 && y < ny - 1 && z < nz - 1;
    R u[3] = {0, 0, 0};
    if (inside && amp != 0.0) startup_velocity<R>((uint64_t)c, seed, amp, u);
    const R v2 = (u[0] * u[0] + u[1] * u[1]) + u[2] * u[2];
    R eq[19];
    equilibria<R>(u[0], u[1], u[2], (R)1.0f - K<R>::k15 * v2, eq);
    S *dd = (S *)d.dd;
#pragma unroll
    for (int i = 0; i < 19; i++) Store<S>::st(dd + opp(i) * d.pstride + c, eq[i], weight<R>(opp(i)));
    d.flags[c] = inside ? (y == ny - 2 ? kLid : kFluid) : kObstacle;
    if (store_v) {
        R *v = (R *)d.vel;
        v[c] = u[0]; v[d.n + c] = u[1]; v[2 * d.n + c] = u[2];
    }
}

}  // namespace lbm
