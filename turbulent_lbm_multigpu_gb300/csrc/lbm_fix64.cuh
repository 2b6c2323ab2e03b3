// lbm_fix64.cuh -- the fluid collision of double populations on the integer
// pipes, bit for bit the IEEE double arithmetic.
//
// GB300's FP64 pipe issues 1.75 lanes per clock and SM (measured, additions,
// products and conversions alike), its integer pipes 64 (shifts, logic,
// multiply-adds) to 128 (additions): one double operation costs as much
// issue time as 40-70 integer ones.  The collision has about 275 of them per
// cell, which bound the double kernels at 9 % of the HBM bandwidth.
//
// Most of them act on numbers of one narrow range.  A flow's populations lie
// within [2^-9, 2^-1), so each is a whole multiple of 2^-61 below 4: an
// integer of 62 bits ("Q61").  On that grid a double addition is an integer
// addition followed by rounding to 53 significant bits, half to even: about
// ten integer operations (Fx).  Moments, pair sums, equilibria (their
// constants 1/18, 1/36, 1/3 are 24-bit floats, so the products need 88 bits)
// and the differences feq - f run that way, the subgrid model's square roots
// and reciprocal in integers of their own; products of two velocities, the
// strain norm and the relaxation's product and sum stay on the FP64 pipe,
// which works beside the integer ones.
//
// Measured (256^3 in 2x2x1 subdomains, subgrid model, per step): 8.39 ms ->
// 3.00 ms (2.00k -> 5.60k MLUPS), 76 double operations per cell instead of
// 275; the FP64 pipe is 65 % busy, the shift and logic pipe 72 %, so that
// neither side has much left to take from the other (the last addition of 4
// to 12 populations moved over here too: 3.08-3.18 ms); 48x40x36 45 -> 19 us,
// 24^3 25 -> 15 us.
//
// Every step rounds as the double operation it stands for, so the results
// are the same bits.  Cells outside the range (populations outside
// [2^-9, 2^-3) moving or [2^-9, 2^-1) at rest, density outside
// [0.875, 1.875), two velocity components of together more than 0.25) are
// refused here and take the double arithmetic.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifndef LBM_HD
#ifdef __CUDACC__
#define LBM_HD __host__ __device__ __forceinline__
#else
#define LBM_HD inline
#endif
#endif

namespace lbm {

LBM_HD uint64_t bits_of(double d) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(d);
#else
    uint64_t b;
    memcpy(&b, &d, 8);
    return b;
#endif
}
LBM_HD double double_of(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)hi, (int)lo);
#else
    const uint64_t b = ((uint64_t)hi << 32) | lo;
    double d;
    memcpy(&d, &b, 8);
    return d;
#endif
}
LBM_HD uint32_t hi32(uint64_t v) { return (uint32_t)(v >> 32); }
LBM_HD uint64_t join(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }
// Position of the highest bit that differs from the sign, -1 if none.
LBM_HD int top_bit(int32_t v) {
#ifdef __CUDA_ARCH__
    int p;
    asm("bfind.s32 %0, %1;" : "=r"(p) : "r"(v));
    return p;
#else
    const uint32_t u = (uint32_t)(v < 0 ? ~v : v);
    return u ? 31 - __builtin_clz(u) : -1;
#endif
}
// Funnel shifts by n in 0..31.
LBM_HD uint32_t shl2(uint32_t lo, uint32_t hi, uint32_t n) {  // high word of (hi:lo) << n
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, n);
#else
    return n ? (hi << n) | (lo >> (32 - n)) : hi;
#endif
}
LBM_HD uint32_t shr2(uint32_t lo, uint32_t hi, uint32_t n) {  // low word of (hi:lo) >> n
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, n);
#else
    return n ? (lo >> n) | (hi << (32 - n)) : lo;
#endif
}
LBM_HD uint64_t mul_wide(uint32_t a, uint32_t b) { return (uint64_t)a * b; }

// Round a Q61 number to 53 significant bits, half to even.  The leading bit
// p of the upper word says how many low bits a double of that size lacks.
LBM_HD int64_t rnd53(int64_t v) {
    const int q = top_bit((int32_t)hi32((uint64_t)v)) - 20;
    const uint32_t k = (uint32_t)(q > 0 ? q : 0);
    const uint32_t m = (1u << k) - 1u;
    const uint32_t odd = ((uint32_t)v >> k) & m & 1u;
    const uint64_t s = (uint64_t)v + (uint64_t)((m >> 1) + odd);
    return (int64_t)join(hi32(s), (uint32_t)s & ~m);
}
// The same for |v| >= 2^-7 (two bits or more to drop) with a sticky bit:
// sticky != 0 says that bits below the grid were dropped from v.
LBM_HD int64_t rnd53_big(int64_t v, uint32_t sticky) {
    const uint32_t k = (uint32_t)(top_bit((int32_t)hi32((uint64_t)v)) - 20);
    const uint32_t m = (1u << k) - 1u;
    const uint32_t odd = (((uint32_t)v >> k) | sticky) & 1u;
    const uint64_t s = (uint64_t)v + (uint64_t)((m >> 1) + odd);
    return (int64_t)join(hi32(s), (uint32_t)s & ~m);
}

// A double on the Q61 grid; + and - are the double operations.
struct Fx {
    int64_t v;
};
LBM_HD Fx operator+(Fx a, Fx b) { return Fx{rnd53(a.v + b.v)}; }
LBM_HD Fx operator-(Fx a, Fx b) { return Fx{rnd53(a.v - b.v)}; }
LBM_HD Fx operator-(Fx a) { return Fx{-a.v}; }
LBM_HD Fx &operator+=(Fx &a, Fx b) { return a = a + b; }
LBM_HD Fx &operator-=(Fx &a, Fx b) { return a = a - b; }

// f in [2^-9, 4).
LBM_HD Fx fx_of(double f) {
    const uint64_t b = bits_of(f);
    const uint32_t hi = hi32(b), lo = (uint32_t)b, s = (hi >> 20) - 1014u;
    const uint32_t m = (hi & 0xFFFFFu) | 0x100000u;
    return Fx{(int64_t)join(shl2(lo, m, s), lo << s)};
}
// The double of a rounded Q61 number v >= 2^-29.
LBM_HD double fx_pos(Fx a) {
    const uint32_t hi = hi32((uint64_t)a.v), lo = (uint32_t)a.v;
    const uint32_t p = (uint32_t)top_bit((int32_t)hi), sh = 31u - p;
    const uint32_t yh = shl2(lo, hi, sh), yl = lo << sh;
    return double_of((yh >> 11) + ((p + 993u) << 20), shr2(yl, yh, 11));
}
// The double of any rounded Q61 number, zero included (+0).
LBM_HD double fx_double(Fx a) {
    const uint32_t s = (uint32_t)((int32_t)hi32((uint64_t)a.v) >> 31);
    const uint64_t u = (uint64_t)(a.v < 0 ? -a.v : a.v);
    const bool small = hi32(u) == 0;  // below 2^-29: the lower word alone
    const uint32_t hi = small ? (uint32_t)u : hi32(u), lo = small ? 0u : (uint32_t)u;
#ifdef __CUDA_ARCH__
    const uint32_t sh = (uint32_t)__clz((int)hi);
#else
    const uint32_t sh = hi ? (uint32_t)__builtin_clz(hi) : 32u;
#endif
    const uint32_t yh = shl2(lo, hi, sh & 31u), yl = lo << (sh & 31u);
    const uint32_t e = (small ? 992u : 1024u) - sh;  // biased exponent less the hidden bit
    const uint32_t h = (yh >> 11) + (e << 20);
    return u == 0 ? 0.0 : double_of(h | (s & 0x80000000u), shr2(yl, yh, 11));
}
// The double product 9/2 s2, s2 in [0, 2^-4), on the Q61 grid: rounded to 53
// bits as the product is, then down to the grid with bit 0 set if bits were
// lost (zero gives 1, less than half of any result's last place).
LBM_HD int64_t fx_half9(double s2) {
    const uint64_t b = bits_of(s2);
    const uint32_t hi = hi32(b), lo = (uint32_t)b;
    const uint64_t l9 = mul_wide(lo, 9u);
    const uint32_t h9 = ((hi & 0xFFFFFu) | 0x100000u) * 9u + hi32(l9);  // 9 times the mantissa: bit 55 or 56 leads
    const uint32_t k = h9 >= 0x01000000u ? 4u : 3u, m = (1u << k) - 1u;
    const uint64_t s = join(h9, (uint32_t)l9) + (uint64_t)((m >> 1) + (((uint32_t)l9 >> k) & 1u));
    const uint32_t sl = (uint32_t)s & ~m;
    const uint32_t mh = shl2(sl, hi32(s), 7), ml = sl << 7;
    // value = (mh:ml) 2^(e - 60), on the grid (mh:ml) >> (-1 - e); e + 1023 = hi >> 20
    uint32_t sh = 1022u - (hi >> 20);
    sh = sh < 63u ? sh : 63u;
    const uint32_t n = sh & 31u;
    const uint32_t a = mh >> n, c = shr2(ml, mh, n);
    const uint32_t lost = (1u << n) - 1u;  // the bits that the shift by n drops
    const bool far = sh >= 32u;
    const uint32_t st = far ? (ml | (mh & lost)) : (ml & lost);
    return (int64_t)join(far ? 0u : a, (far ? a : c) | (st ? 1u : 0u));
}
// The double product of a rounded Q61 number in (0, 4) and C 2^-N (C of 24
// bits), for results of at least 2^-7.
template <uint32_t C, uint32_t N>
LBM_HD Fx fx_times(Fx a) {
    const uint64_t l = mul_wide((uint32_t)a.v, C);
    const uint64_t h = mul_wide(hi32((uint64_t)a.v), C) + hi32(l);
    const uint32_t low = (uint32_t)l, lost = low & ((1u << N) - 1u);
    return Fx{rnd53_big((int64_t)join(shr2((uint32_t)h, hi32(h), N), shr2(low, (uint32_t)h, N)), lost ? 1u : 0u)};
}
// The reference's float constants as C 2^-N.
LBM_HD Fx fx_c18(Fx a) { return fx_times<14913081u, 28>(a); }
LBM_HD Fx fx_c36(Fx a) { return fx_times<14913081u, 29>(a); }
LBM_HD Fx fx_c3(Fx a) { return fx_times<11184811u, 25>(a); }
static_assert((float)(14913081.0 / 268435456.0) == 1.0f / 18.0f && (float)(14913081.0 / 536870912.0) == 1.0f / 36.0f &&
                  (float)(11184811.0 / 33554432.0) == 1.0f / 3.0f,
              "24-bit forms of the equilibrium constants");

// The opposite pair of equilibria r +- 3 s + 9/2 s^2 (before the constant).
LBM_HD void fx_pair(Fx r, Fx s, double s2, Fx &p, Fx &m) {
    const Fx t{rnd53(s.v + s.v + s.v)};
    const int64_t z = fx_half9(s2);
    p = Fx{rnd53_big(rnd53_big(r.v + t.v, 0u) + z, 0u)};
    m = Fx{rnd53_big(rnd53_big(r.v - t.v, 0u) + z, 0u)};
}

// Whether populations lie within the range: every moving one in [2^-9, 2^-3),
// the one at rest in [2^-9, 2^-1).
LBM_HD bool fx_ordinary(const double f[19]) {
    uint32_t out = 0;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int i = 0; i < 18; i++) {
        const uint32_t u = hi32(bits_of(f[i])) - 0x3F600000u;
        out = out > u ? out : u;
    }
    return out < 0x00600000u && hi32(bits_of(f[18])) - 0x3F600000u < 0x00800000u;
}
// Density in [0.875, 1.875), and sums and differences of any two velocity
// components within 0.25 (to a unit of 2^-29, the upper words' last place).
// The equilibria need |s| <= 0.25 for every direction's s = e.u: then d = r -
// 3/2 u^2 is 0.78 or more, d - 3 s at least 2^-7, no equilibrium below 2^-7, and
// 9/2 s^2 and the sums stay within their formats.  (Components below 0.125
// each, the bound at first, sent flows of 0.125 to 0.25 along an axis to the
// double arithmetic and warps with some such cells both ways: 128^3 at 0.15,
// 1,281 us per step, 1,051 in double arithmetic alone, 593 now; 48x40x36 73, 46 and
// 45.)  In this form both units' kernels compile with no more spills than
// under the narrower bound; with magnitudes and a minimum, beta spilled twice
// as much.
LBM_HD bool fx_flow(Fx r, Fx vx, Fx vy, Fx vz) {
    const auto small = [](uint32_t h) { return h + 0x08000000u < 0x0FFFFFFFu; };
    const uint32_t x = hi32((uint64_t)vx.v), y = hi32((uint64_t)vy.v), z = hi32((uint64_t)vz.v);
    return hi32((uint64_t)r.v) - 0x1C000000u < 0x20000000u && small(x + y) && small(x - y) && small(x + z) &&
           small(x - z) && small(y + z) && small(y - z);
}

// Estimates of 1/sqrt(x) and 1/x to about 2^-22 (any better one does).
LBM_HD float rsqrt_estimate(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / sqrtf(x);
#endif
}
LBM_HD float rcp_estimate(float x) {
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}
LBM_HD float float_of(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, 4);
    return f;
#endif
}
LBM_HD uint32_t float_bits(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t b;
    memcpy(&b, &f, 4);
    return b;
#endif
}
// Nearest integer of a float below 2^31 in magnitude (ties either way).
LBM_HD int32_t near_int(float f) {
#ifdef __CUDA_ARCH__
    return __float2int_rn(f);
#else
    return (int32_t)lrintf(f);
#endif
}

// The square root and the reciprocal of a double, correctly rounded, in
// integers.  A float estimate (24 bits) is refined twice by its exact
// remainder, known modulo 2^64 and small (Newton's iteration, 46 and 63
// bits); the last bit is settled by the sign of the exact remainder at the
// midpoint between the two candidates (Tuckerman's test).
//
// x in [2^-120, 2^100].
LBM_HD double sqrt_int(double x) {
    const uint64_t b = bits_of(x);
    const uint32_t hi = hi32(b), lo = (uint32_t)b;
    // x = X 2^(2 j - 62), X in [2^60, 2^62): mantissa bit 52 moves to bit 60 (odd exponent: 61)
    const uint32_t ex = hi >> 20;          // biased exponent e + 1023
    const uint32_t odd = (ex & 1u) ^ 1u;   // e odd
    const uint32_t m = (hi & 0xFFFFFu) | 0x100000u;
    const uint64_t X = join(shl2(lo, m, 8u + odd), lo << (8u + odd));
    // m' = X 2^-62 in [2^-2, 1); y ~ 1/sqrt(m') in (1, 2]
    const float mf = float_of(((odd ? 126u : 125u) << 23) | shl2(lo, m & 0xFFFFFu, 3));
    const float y = rsqrt_estimate(mf);
    const uint32_t s0 = (uint32_t)near_int(mf * y * 16777216.0f);             // sqrt(m') 2^24
    const int64_t r0 = (int64_t)(X - (mul_wide(s0, s0) << 14));               // |r0| < 2^42
    const int32_t d0 = near_int((float)(int32_t)(r0 >> 12) * y * 0x1p-4f);    // r0 / (2 sqrt) 2^(47 - 62)
    const uint64_t s1 = ((uint64_t)s0 << 23) + (uint64_t)(int64_t)d0;         // sqrt(m') 2^47
    const int64_t r1 = (int64_t)((X << 32) - s1 * s1);                        // |r1| < 2^54
    const int32_t d1 = near_int((float)(int32_t)(r1 >> 24) * y * 0x1p-8f);    // r1 / (2 sqrt) 2^(63 - 94)
    const uint64_t s2 = (s1 << 16) + (uint64_t)(int64_t)d1;                   // sqrt(m') 2^63
    const uint64_t c = s2 >> 10, h = 2 * c + 1;                               // midpoint above c, 54 bits
    const uint64_t r = c + ((int64_t)((X << 46) - h * h) > 0 ? 1u : 0u);
    // r has its leading one at bit 52, which adds 1 to the exponent field; the
    // result's exponent is floor(e / 2)
    return double_of(hi32(r) + ((((ex + 1023u) >> 1) - 1u) << 20), (uint32_t)r);
}
// x in [2^-60, 2^60].
LBM_HD double rcp_int(double x) {
    const uint64_t b = bits_of(x);
    const uint32_t hi = hi32(b), lo = (uint32_t)b;
    const uint64_t t = join((hi & 0xFFFFFu) | 0x100000u, lo);                 // mantissa in [2^52, 2^53)
    const float mf = float_of((127u << 23) | shl2(lo, hi & 0xFFFFFu, 3));     // in [1, 2)
    const float y = rcp_estimate(mf);
    const uint32_t y0 = (uint32_t)near_int(y * 16777216.0f);                  // 2^76 / t
    const int64_t r0 = (int64_t)(0 - t * y0);                                 // 2^76 - t y0, |r0| < 2^56
    const int32_t d0 = near_int((float)(int32_t)(r0 >> 26) * y * 0x1p-3f);    // r0 2^23 / t
    const uint64_t y1 = ((uint64_t)y0 << 23) + (uint64_t)(int64_t)d0;         // 2^99 / t
    const int64_t r1 = (int64_t)(0 - t * y1);                                 // 2^99 - t y1, |r1| < 2^58
    const int32_t d1 = near_int((float)(int32_t)(r1 >> 28) * y * 0x1p-8f);    // r1 2^16 / t
    const uint64_t y2 = (y1 << 16) + (uint64_t)(int64_t)d1;                   // 2^115 / t
    const uint64_t c = y2 >> 10, h = 2 * c + 1;
    const uint64_t r = c + ((int64_t)(0 - t * h) > 0 ? 1u : 0u);              // 2^105 / t in (2^52, 2^53]
    return double_of(hi32(r) + ((2044u - (hi >> 20)) << 20), (uint32_t)r);
}

LBM_HD double fx_sqrt(double x) {
    return hi32(bits_of(x)) - 0x38700000u < 0x0DC00000u ? sqrt_int(x) : sqrt(x);  // [2^-120, 2^100)
}

// Whether the parameters are ones fx_collide reproduces for every ordinary
// cell: a finite rate, and with the subgrid model a coefficient and a tau0
// whose sum of roots stays within rcp_int's range (the strain norm q of
// ordinary populations is below 2^5).  Others (negative, huge, infinite, not a
// number) take the double arithmetic.
LBM_HD bool fx_params(double inv_tau, double tau0, double les_c) {
    if (les_c == 0.0) return inv_tau - inv_tau == 0.0;
    return les_c > 0.0 && les_c <= 0x1p100 && tau0 >= 0.5 && tau0 <= 0x1p50;
}

// The collision of an ordinary fluid cell from its moments on the grid, under
// parameters that fx_params accepts (operation by operation that of collide()): populations x in, f out; vx,
// vy, vz and dp come out as doubles.
template <bool LES>
LBM_HD void fx_collide(const Fx x[19], Fx r, Fx jx, Fx jy, Fx jz, double inv_tau, double tau0, double les_c, double f[19],
                       double &dp, double &vx, double &vy, double &vz) {
    vx = fx_double(jx);
    vy = fx_double(jy);
    vz = fx_double(jz);
    const double xx = vx * vx, yy = vy * vy, zz = vz * vz;
    const double rho = fx_pos(r);
    dp = rho - 1.5 * ((xx + yy) + zz);
    double w = inv_tau;
    if (LES && les_c != 0.0) {
        Fx p[9];
#ifdef __CUDACC__
#pragma unroll
#endif
        for (int k = 0; k < 9; k++) p[k] = x[2 * k] + x[2 * k + 1];
        const Fx sxx = (((p[0] + p[2]) + p[3]) + p[4]) + p[5];
        const Fx syy = (((p[1] + p[2]) + p[3]) + p[6]) + p[7];
        const Fx szz = (((p[4] + p[5]) + p[6]) + p[7]) + p[8];
        const Fx r3 = fx_c3(r);
        const double pxx = fx_double(sxx - r3) - xx;
        const double pyy = fx_double(syy - r3) - yy;
        const double pzz = fx_double(szz - r3) - zz;
        const double pxy = fx_double(p[2] - p[3]) - vx * vy;
        const double pxz = fx_double(p[4] - p[5]) - vx * vz;
        const double pyz = fx_double(p[6] - p[7]) - vy * vz;
        // twice the second sum is exact, so it may fuse
        const double q = fma(2.0, (pxy * pxy + pxz * pxz) + pyz * pyz, (pxx * pxx + pyy * pyy) + pzz * pzz);
        const double g = tau0 * tau0 + les_c * fx_sqrt(q);
        const double te2 = tau0 + fx_sqrt(g);
        // 1 / (te2 / 2): the halved exponent is exact
        const uint64_t b = bits_of(te2);
        w = rcp_int(double_of(hi32(b) - 0x100000u, (uint32_t)b));
    }
    const Fx d = fx_of(dp);
    // f += w (feq - f).  A difference |D| 2^-61 below 2^-9 (|D| < 2^52) needs
    // no rounding, and as the low bits of a double it is 2^-9 + |D| 2^-61: w
    // times that less w 2^-9 (exact) is the rounded product in one fused
    // operation, without normalising D.  A larger one has its leading bit at
    // 20 or above in the upper word; it is rounded and shifted there.
    const double wb = w * -0x1p-9;
    const auto relax = [&](int i, Fx e) {
        const int64_t D = e.v - x[i].v;
        const uint64_t a = (uint64_t)(D < 0 ? -D : D);
        const uint32_t sign = hi32((uint64_t)D) & 0x80000000u;
        const bool big = hi32(a) >= 0x100000u;
        const int q = top_bit((int32_t)hi32(a)) - 20;
        const uint32_t k = (uint32_t)(q > 0 ? q : 0), m = (1u << k) - 1u;
        const uint64_t g = a + (uint64_t)((m >> 1) + (((uint32_t)a >> k) & m & 1u));
        const double t = double_of((hi32(g) >> k) + ((big ? 0x3F5u + k : 0x3F6u) << 20), shr2((uint32_t)g, hi32(g), k));
        const double sw = double_of(hi32(bits_of(w)) ^ sign, (uint32_t)bits_of(w));
        const double sb = big ? 0.0 : double_of(hi32(bits_of(wb)) ^ sign, (uint32_t)bits_of(wb));
        f[i] = fx_pos(x[i]) + fma(sw, t, sb);
    };
    const auto axis = [&](int k, Fx s, double s2) {
        Fx p, m;
        fx_pair(d, s, s2, p, m);
        relax(2 * k, fx_c18(p));
        relax(2 * k + 1, fx_c18(m));
    };
    const auto diag = [&](int k, Fx s) {
        const double v = fx_double(s);
        Fx p, m;
        fx_pair(d, s, v * v, p, m);
        relax(2 * k, fx_c36(p));
        relax(2 * k + 1, fx_c36(m));
    };
    axis(0, jx, xx);
    axis(1, jy, yy);
    diag(2, jx + jy);
    diag(3, jx - jy);
    diag(4, jx + jz);
    diag(5, jx - jz);
    diag(6, jy + jz);
    diag(7, jy - jz);
    axis(8, jz, zz);
    relax(18, fx_c3(d));
}

// The equilibria of a lid cell (vy = vz = 0): populations f and dd_param.
// The lid speed has to lie on the grid below 0.125: a magnitude in [2^-9,
// 2^-3) or zero.
LBM_HD bool fx_lid_speed(double lid) {
    return lid == 0.0 || (hi32(bits_of(lid)) & 0x7FFFFFFFu) - 0x3F600000u < 0x00600000u;
}
LBM_HD void fx_lid(double lid, double f[19], double &dp) {
    const double xx = lid * lid;
    dp = 1.0 - 1.5 * xx;
    const Fx d = fx_of(dp), zero{0};
    Fx s = zero;
    if (lid != 0.0) s = fx_of(fabs(lid));
    if (lid < 0.0) s = -s;
    Fx p, m;
    fx_pair(d, s, xx, p, m);
    f[0] = fx_pos(fx_c18(p));
    f[1] = fx_pos(fx_c18(m));
    const double ep = fx_pos(fx_c36(p)), em = fx_pos(fx_c36(m));
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 2; k < 6; k++) {  // directions with an x component
        f[2 * k] = ep;
        f[2 * k + 1] = em;
    }
    f[2] = f[3] = f[16] = f[17] = fx_pos(fx_c18(d));
    f[12] = f[13] = f[14] = f[15] = fx_pos(fx_c36(d));
    f[18] = fx_pos(fx_c3(d));
}

// ------------------------------------------------- without the roundings
// The contracted double kernels need not reproduce the roundings of the
// double operations, only stay as close to the model: on the grid, sums are
// exact, products are cut at 2^-61 (a double population's last place is
// 2^-57 to 2^-59), and only the new population rounds to 53 bits.  About 10
// double operations per cell remain, in the strain norm.  Measured (256^3 in
// 2x2x1 subdomains, subgrid model): 6.14 -> 1.64 ms per step (10.2k MLUPS) at
// 2 blocks of 256 per SM (128 registers; 3 blocks spill more and take 1.86,
// 4 blocks 2.55), 1,940-2,000 instructions per cell, the shift and logic pipe
// 60 % busy.

// High half of the signed 128-bit product.
LBM_HD int64_t mul_high(int64_t a, int64_t b) {
#ifdef __CUDA_ARCH__
    return __mul64hi(a, b);
#else
    return (int64_t)(((__int128)a * b) >> 64);
#endif
}
// v C 2^-N rounded to the grid, v in (0, 4).
template <uint32_t C, uint32_t N>
LBM_HD int64_t fq_times(int64_t v) {
    const uint64_t l = mul_wide((uint32_t)v, C) + (1u << (N - 1));
    const uint64_t h = mul_wide(hi32((uint64_t)v), C) + hi32(l);
    return (int64_t)join(shr2((uint32_t)h, hi32(h), N), shr2((uint32_t)l, (uint32_t)h, N));
}
// The double nearest to a grid number v >= 2^-29.
LBM_HD double fq_pos(int64_t v) {
    const uint32_t hi = hi32((uint64_t)v), lo = (uint32_t)v;
    const uint32_t p = (uint32_t)top_bit((int32_t)hi), sh = 31u - p;
    const uint32_t yh = shl2(lo, hi, sh), yl = lo << sh;
    const uint64_t m = join((yh >> 11) + ((p + 993u) << 20), shr2(yl, yh, 11)) + ((yl >> 10) & 1u);
    return double_of(hi32(m), (uint32_t)m);
}

// The collision of an ordinary fluid cell: populations x on the grid in, f
// out, and where asked for (out) the velocity, the density m and dd_param.
// False: the cell is out of range (or its relaxation rate or a result is), f
// is not the result.
template <bool LES>
LBM_HD bool fq_collide(const Fx x[19], double inv_tau, double tau0, double les_c, bool out, double f[19], double &m,
                       double &dp, double &vx, double &vy, double &vz) {
    int64_t p[9], t[9];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 0; k < 9; k++) {
        p[k] = x[2 * k].v + x[2 * k + 1].v;
        t[k] = x[2 * k].v - x[2 * k + 1].v;
    }
    const int64_t a23 = p[2] + p[3], a45 = p[4] + p[5], a67 = p[6] + p[7];
    const Fx r{p[0] + p[1] + p[8] + x[18].v + a23 + a45 + a67};
    const Fx jx{t[0] + t[2] + t[3] + t[4] + t[5]}, jy{t[1] + t[2] - t[3] + t[6] + t[7]},
        jz{t[4] - t[5] + t[6] - t[7] + t[8]};
    if (!fx_flow(r, jx, jy, jz)) return false;
    // products of velocities in units of 2^-64
    const int64_t ux = jx.v << 3, uy = jy.v << 3, uz = jz.v << 3;
    const int64_t xx = mul_high(ux, ux), yy = mul_high(uy, uy), zz = mul_high(uz, uz);
    const int64_t xy = mul_high(ux, uy), xz = mul_high(ux, uz), yz = mul_high(uy, uz);
    const int64_t d = r.v - ((3 * (xx + yy + zz)) >> 4);
    if (out) {
        m = fq_pos(r.v);
        dp = fq_pos(d);
        vx = fx_double(jx);
        vy = fx_double(jy);
        vz = fx_double(jz);
    }
    double w = inv_tau;
    if (LES && les_c != 0.0) {
        const int64_t r3 = fq_times<11184811u, 25>(r.v);
        const double pxx = fx_double(Fx{(p[0] + a23 + a45 - r3) - (xx >> 3)});
        const double pyy = fx_double(Fx{(p[1] + a23 + a67 - r3) - (yy >> 3)});
        const double pzz = fx_double(Fx{(p[8] + a45 + a67 - r3) - (zz >> 3)});
        const double pxy = fx_double(Fx{(p[2] - p[3]) - (xy >> 3)});
        const double pxz = fx_double(Fx{(p[4] - p[5]) - (xz >> 3)});
        const double pyz = fx_double(Fx{(p[6] - p[7]) - (yz >> 3)});
        const double q = fma(2.0, fma(pyz, pyz, fma(pxz, pxz, pxy * pxy)), fma(pzz, pzz, fma(pyy, pyy, pxx * pxx)));
        const double te2 = tau0 + fx_sqrt(fma(les_c, fx_sqrt(q), tau0 * tau0));
        const uint64_t b = bits_of(te2);
        w = rcp_int(double_of(hi32(b) - 0x100000u, (uint32_t)b));
    }
    // w in [2^-9, 2) in units of 2^-62
    const uint32_t wh = hi32(bits_of(w));
    if (wh - 0x3F600000u >= 0x00A00000u) return false;
    const int64_t wi = fx_of(w).v << 1;
    int32_t low = 0x7FFFFFFF;  // smallest upper word of the results
    const auto relax = [&](int i, int64_t e) {
        const int64_t n = x[i].v + mul_high((e - x[i].v) << 2, wi);
        const int32_t h = (int32_t)hi32((uint64_t)n);
        low = low < h ? low : h;
        f[i] = fq_pos(n);
    };
    const auto axis = [&](int k, Fx s, int64_t s2) {
        const int64_t q = d + ((4 * s2 + (s2 >> 1)) >> 3), o = 3 * s.v;
        relax(2 * k, fq_times<14913081u, 28>(q + o));
        relax(2 * k + 1, fq_times<14913081u, 28>(q - o));
    };
    const auto diag = [&](int k, int64_t s, int64_t s2) {
        const int64_t q = d + ((4 * s2 + (s2 >> 1)) >> 3), o = 3 * s;
        relax(2 * k, fq_times<14913081u, 29>(q + o));
        relax(2 * k + 1, fq_times<14913081u, 29>(q - o));
    };
    axis(0, jx, xx);
    axis(1, jy, yy);
    diag(2, jx.v + jy.v, xx + yy + 2 * xy);
    diag(3, jx.v - jy.v, xx + yy - 2 * xy);
    diag(4, jx.v + jz.v, xx + zz + 2 * xz);
    diag(5, jx.v - jz.v, xx + zz - 2 * xz);
    diag(6, jy.v + jz.v, yy + zz + 2 * yz);
    diag(7, jy.v - jz.v, yy + zz - 2 * yz);
    axis(8, jz, zz);
    relax(18, fq_times<11184811u, 25>(d));
    return low >= 0x00010000;  // 2^-13: the grid is 2^-48 of the smallest result
}

}  // namespace lbm
