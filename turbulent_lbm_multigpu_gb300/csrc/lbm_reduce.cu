// lbm_reduce.cu -- conservation sums and velocity errors of resident lattices.
//
// Both quantities are sums over the fluid cells of moments of the stored
// populations, asked for in (better than) FP64.  GB300's FP64 pipe issues
// about 1.75 lanes per clock and SM (measured; conversions between float and
// double run on it too), so sums written in double arithmetic are bound by
// that pipe: 19 conversions, 45 additions and the compensated accumulation
// took 5.0 ms for a 256^3 half lattice whose bytes take 0.1 ms to read.
//
// The populations of a flow are fixed-point numbers in all but name: the
// moving ones lie within [2^-8, 2^-3), the one at rest within [2^-8, 2^-1)
// (|u| below 0.3), so a float one is a whole multiple of 2^-31 and a double
// one (from 2^-9) of 2^-61.  Cells within those bounds are summed exactly in
// integers: moments in 32 (64) bits, squares of the momentum in 64 (128),
// totals in 128 and those of double cells' squares in 160 (Squares).  The sums
// then do not depend on the order of the cells and round once, at the end.  A cell with any population outside the bounds
// (negative, large, infinite, not a number) is summed in double arithmetic
// with compensation, as the whole lattice was before.
//
// Measured (256^3 cavity, whole calls): sums of a half lattice 5.4 -> 0.24 ms,
// of a double one 4.8 -> 0.45 ms (5.7 TB/s), velocity error of half against
// double 7.2 -> 0.56 ms (5.7 TB/s); the final stages, one thread per quantity
// before, 0.33-0.38 ms -> 5 us.
#include <algorithm>
#include <mutex>
#include <string>

#include "lbm_internal.h"

using namespace lbm;
using namespace lbm_rt;

namespace {
typedef __int128 i128;
typedef unsigned __int128 u128;

// Neumaier-compensated FP64 accumulation.
struct Acc {
    double s, c;
    __device__ __forceinline__ void add(double v) {
        const double t = s + v;
        if (fabs(s) >= fabs(v)) c += (s - t) + v;
        else c += (v - t) + s;
        s = t;
    }
    __device__ __forceinline__ void merge(const Acc &o) {
        add(o.s);
        c += o.c;
    }
};

// Fixed-point moments of one cell.  mass and j come in units of 2^-kLsb;
// returns false when a population lies outside the bounds (the values are
// then meaningless).  j belongs to slot order; the opposite order negates it.
template <typename R> struct CellFix;
template <> struct CellFix<float> {
    static constexpr int kLsb = 31;
    using J = int32_t;  // |j| < 5 * 2^-3 < 1
    __device__ static __forceinline__ bool of(const float f[19], uint64_t &mass, J j[3]) {
        uint32_t v[19], out = 0;
#pragma unroll
        for (int i = 0; i < 19; i++) {
            v[i] = __float2uint_rz(f[i] * 0x1p31f);
            if (i < 18) out = max(out, __float_as_uint(f[i]) - 0x3B800000u);  // 2^-8
        }
        const uint32_t rest = __float_as_uint(f[18]) - 0x3B800000u;
        sums(v, j);
        uint32_t a = 0, b = v[18];  // 9 and 10 populations: below 2^32 each
#pragma unroll
        for (int i = 0; i < 9; i++) {
            a += v[i];
            b += v[i + 9];
        }
        mass = (uint64_t)a + b;
        return out < 0x02800000u && rest < 0x03800000u;  // 2^-3, 2^-1
    }
    template <typename T, typename U> __device__ static __forceinline__ void sums(const U v[19], T j[3]) {
        U s[3] = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < 18; i++) {
            s[0] += dir_x(i) > 0 ? v[i] : dir_x(i) < 0 ? (U)0 - v[i] : (U)0;
            s[1] += dir_y(i) > 0 ? v[i] : dir_y(i) < 0 ? (U)0 - v[i] : (U)0;
            s[2] += dir_z(i) > 0 ? v[i] : dir_z(i) < 0 ? (U)0 - v[i] : (U)0;
        }
#pragma unroll
        for (int a = 0; a < 3; a++) j[a] = (T)s[a];
    }
};
template <> struct CellFix<double> {
    static constexpr int kLsb = 61;
    using J = int64_t;
    __device__ static __forceinline__ bool of(const double f[19], uint64_t &mass, J j[3]) {
        uint64_t v[19];
        uint32_t out = 0, rest = 0;
        mass = 0;
#pragma unroll
        for (int i = 0; i < 19; i++) {
            const uint32_t hi = (uint32_t)__double2hiint(f[i]), lo = (uint32_t)__double2loint(f[i]);
            const uint32_t u = hi - 0x3F600000u;  // 2^-9
            if (i < 18) out = max(out, u);
            else rest = u;
            v[i] = ((((uint64_t)((hi & 0xFFFFFu) | 0x100000u)) << 32) | lo) << ((u >> 20) & 31u);
            mass += v[i];
        }
        CellFix<float>::sums(v, j);
        return out < 0x00600000u && rest < 0x00800000u;  // 2^-3, 2^-1
    }
};

__device__ __forceinline__ u128 square(int64_t v) {
    const uint64_t a = (uint64_t)(v < 0 ? -v : v);
    return ((u128)__umul64hi(a, a) << 64) | (a * a);
}

__device__ __forceinline__ i128 shfl_down(i128 v, int o) {
    const u128 u = (u128)v;
    const uint64_t lo = __shfl_down_sync(0xffffffffu, (unsigned long long)u, o);
    const uint64_t hi = __shfl_down_sync(0xffffffffu, (unsigned long long)(u >> 64), o);
    return (i128)(((u128)hi << 64) | lo);
}
__device__ __forceinline__ i128 warp_sum(i128 v) {
    for (int o = 16; o > 0; o >>= 1) v += shfl_down(v, o);
    return v;
}
__device__ __forceinline__ i128 warp_max(i128 v) {
    for (int o = 16; o > 0; o >>= 1) {
        const i128 w = shfl_down(v, o);
        v = w > v ? w : v;
    }
    return v;
}
__device__ __forceinline__ uint64_t warp_sum(uint64_t v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, (unsigned long long)v, o);
    return v;
}
// The double nearest to (v + low 2^-32) 2^-lsb; low only where v >= 0.
__device__ double to_double(i128 v, int lsb, uint32_t low = 0) {
    const bool neg = v < 0;
    u128 m = neg ? (u128)0 - (u128)v : (u128)v;
    if (m >> 96) {
        m |= low ? 1 : 0;  // far below the last place of a double
    } else {
        m = (m << 32) | low;
        lsb += 32;
    }
    if (m == 0) return 0.0;
    const uint64_t hi = (uint64_t)(m >> 64);
    const int s = hi ? __clzll((long long)hi) : 64 + __clzll((long long)(uint64_t)m);
    m <<= s;
    // 64 leading bits, the last one set if any below is: one rounding, here
    const double d = scalbn(__ull2double_rn((uint64_t)(m >> 64) | ((uint64_t)m ? 1u : 0u)), 64 - s - lsb);
    return neg ? -d : d;
}

// Exact total of squares in units of 2^-122 (each below 2^125): the upper 96
// bits of each in one sum (units of 2^-90), the lower 32 in another, so that
// 2^31 cells of any size fit and the smallest count.  LOW false: the
// squares are whole multiples of 2^-90 (float cells).
template <bool LOW> struct Squares {
    i128 hi = 0;
    uint64_t lo = 0;
    __device__ __forceinline__ void add(u128 e) {
        hi += (i128)(e >> 32);
        if (LOW) lo += (uint32_t)e;
    }
};

// Partial results of a block: five exact sums and five compensated ones
// (cells outside the fixed-point bounds).
struct RedPartial {
    i128 fix[5];
    Acc acc[5];
    uint64_t low;  // of the energy's squares (Squares::lo)
};
// Blocks of a reduction: a few per SM; every thread walks the lattice with
// the stride of the whole grid.
constexpr int kRedBlocks = 1024;
static_assert(kRedBlocks * sizeof(RedPartial) <= 256 * 1024, "partials of a reduction");

// Cells c..c+V-1 of a lattice, populations as stored values of R.
template <typename S, int V> struct Cells {
    using R = typename Store<S>::R;
    R f[V][19];
    __device__ __forceinline__ void load(const LatDesc &d, int64_t c) {
        const S *p = (const S *)d.dd + c;
#pragma unroll
        for (int i = 0; i < 19; i++) {
            if constexpr (V == 2) {
                const P2 v = Store<S>::ld2(p + i * d.pstride, weight<R>(i));
                f[0][i] = v.x;
                f[1][i] = v.y;
            } else {
                f[0][i] = Store<S>::ld(p + i * d.pstride, weight<R>(i));
            }
        }
    }
};

// Moments of a cell in double arithmetic (any values).  Rolled up: it runs
// for few cells, and unrolled it would hold registers of the common path.
template <typename R>
__device__ __forceinline__ void moments_double(const R f[19], double &r, double j[3]) {
    R t[19];
#pragma unroll
    for (int i = 0; i < 19; i++) t[i] = f[i];
    r = j[0] = j[1] = j[2] = 0.0;
#pragma unroll 1
    for (int i = 0; i < 19; i++) {
        const double v = (double)t[i];
        r += v;
        j[0] += dir_x(i) * v;
        j[1] += dir_y(i) * v;
        j[2] += dir_z(i) * v;
    }
}

// Sums of mass, momentum and kinetic energy over the fluid cells.  Float and
// 16-bit lattices take two cells per thread (wider loads: 19 of 8 or 4 bytes
// in flight per thread), double ones one.
template <typename S>
__global__ void __launch_bounds__(kBlock, 2) k_reduce(LatDesc d, int layout, RedPartial *partial) {
    using R = typename Store<S>::R;
    using F = CellFix<R>;
    constexpr int V = sizeof(R) == 4 ? 2 : 1;
    __shared__ Acc sh[5][kBlock];
    __shared__ i128 wsum[kBlock / 32][5];
    __shared__ uint64_t wlow[kBlock / 32];
    constexpr bool kLow = sizeof(R) == 8;
    i128 tot[5] = {0, 0, 0, 0, 0};
    uint64_t low = 0;
    bool odd = false;  // this thread has summed a cell in double arithmetic
    for (int64_t c = V * ((int64_t)blockIdx.x * kBlock + threadIdx.x); c < d.n; c += (int64_t)V * gridDim.x * kBlock) {
        // planes and flags are padded beyond n (256 bytes): a pair may read past the last cell
        const int fl = V == 2 ? *(const uint16_t *)(d.flags + c) : d.flags[c];
        const bool on[2] = {(fl & 0xff) == kFluid, V == 2 && (fl >> 8) == kFluid && c + 1 < d.n};
        if (!on[0] && !on[1]) continue;
        Cells<S, V> q;
        q.load(d, c);
#pragma unroll
        for (int h = 0; h < V; h++) {
            if (!on[h]) continue;
            uint64_t mass;
            typename F::J j[3];
            if (F::of(q.f[h], mass, j)) {
                tot[0] += mass;
                for (int a = 0; a < 3; a++) tot[1 + a] += j[a];
                if constexpr (sizeof(R) == 4) {
                    uint64_t e = 0;  // units of 2^-62
                    for (int a = 0; a < 3; a++) e += (uint64_t)((int64_t)j[a] * j[a]);
                    tot[4] += e;
                } else {
                    u128 e = 0;  // units of 2^-122
                    for (int a = 0; a < 3; a++) e += square(j[a]);
                    tot[4] += (i128)(e >> 32);
                    low += (uint32_t)e;
                }
            } else {
                if (!odd)
                    for (int k = 0; k < 5; k++) sh[k][threadIdx.x] = Acc{0.0, 0.0};
                odd = true;
                double r, m[3];
                moments_double<R>(q.f[h], r, m);
                sh[0][threadIdx.x].add(r);
                for (int a = 0; a < 3; a++) sh[1 + a][threadIdx.x].add(layout ? -m[a] : m[a]);
                sh[4][threadIdx.x].add(0.5 * (m[0] * m[0] + m[1] * m[1] + m[2] * m[2]));
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = 0; k < 5; k++) {
        const i128 v = warp_sum(tot[k]);
        if (lane == 0) wsum[warp][k] = v;
    }
    if constexpr (kLow) {
        low = warp_sum(low);
        if (lane == 0) wlow[warp] = low;
    }
    if (__syncthreads_or(odd)) {
        if (!odd)
            for (int k = 0; k < 5; k++) sh[k][threadIdx.x] = Acc{0.0, 0.0};
        __syncthreads();
        for (int w = kBlock / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w)
                for (int k = 0; k < 5; k++) sh[k][threadIdx.x].merge(sh[k][threadIdx.x + w]);
            __syncthreads();
        }
    } else if (threadIdx.x < 5) {
        sh[threadIdx.x][0] = Acc{0.0, 0.0};
    }
    if (threadIdx.x < 5) {
        i128 v = 0;
        for (int w = 0; w < kBlock / 32; w++) v += wsum[w][threadIdx.x];
        partial[blockIdx.x].fix[threadIdx.x] = layout && threadIdx.x >= 1 && threadIdx.x <= 3 ? -v : v;
        partial[blockIdx.x].acc[threadIdx.x] = sh[threadIdx.x][0];
    } else if (threadIdx.x == 5) {
        uint64_t v = 0;
        if (kLow)
            for (int w = 0; w < kBlock / 32; w++) v += wlow[w];
        partial[blockIdx.x].low = v;
    }
}

// Final stage: warp q sums quantity q of all blocks, a lane per strided
// share.  lsb: units of mass and momentum, lsb_e of the energy's j^2.
__global__ void __launch_bounds__(160) k_reduce_final(const RedPartial *partial, int nblocks, int lsb, int lsb_e,
                                                      double *out) {
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    i128 v = 0;
    uint64_t low = 0;
    Acc a{0.0, 0.0};
#pragma unroll 4
    for (int b = lane; b < nblocks; b += 32) {
        v += partial[b].fix[q];
        if (q == 4) low += partial[b].low;
        const Acc o = partial[b].acc[q];
        if (!(o.s == 0.0 && o.c == 0.0)) a.merge(o);
    }
    v = warp_sum(v);
    low = warp_sum(low);
    v += (i128)(low >> 32);
    for (int o = 16; o > 0; o >>= 1) {
        const Acc other{__shfl_down_sync(0xffffffffu, a.s, o), __shfl_down_sync(0xffffffffu, a.c, o)};
        if (lane + o < 32) a.merge(other);
    }
    if (lane == 0) {
        a.add(q == 4 ? 0.5 * to_double(v, lsb_e, (uint32_t)low) : to_double(v, lsb));
        out[q] = a.s + a.c;
    }
}

// Velocity difference of two lattices of the same size over the fluid cells
// of `a`: max |ua - ub|, sum |ua - ub|^2, sum |ub|^2, max |ub|, cell count,
// with u the momentum of the stored populations in the given slot layouts.
// Momenta in units of 2^-61, squares of 2^-122, their sums of 2^-90 and the
// lower words' (Squares).
struct CmpPartial {
    i128 fix[4];  // max |ua - ub|^2, its sum, sum |ub|^2, max |ub|^2
    double acc[4];  // the same of cells outside the fixed-point bounds: max, sum, sum, max
    uint64_t low[2];  // lower words of the two sums
    double cells;
    double pad;
};
static_assert(sizeof(CmpPartial) <= sizeof(RedPartial), "one workspace for both reductions");

template <typename SA, typename SB>
__global__ void __launch_bounds__(kBlock, 2) k_compare(LatDesc a, int la, LatDesc b, int lb, CmpPartial *partial) {
    using RA = typename Store<SA>::R;
    using RB = typename Store<SB>::R;
    __shared__ double sh[4][kBlock];
    __shared__ i128 wred[kBlock / 32][5];
    __shared__ uint64_t wlow[kBlock / 32][2];
    i128 mx = 0, mr = 0;
    Squares<sizeof(RA) == 8 || sizeof(RB) == 8> se;
    Squares<sizeof(RB) == 8> sr;
    uint32_t cnt = 0;
    double dv[4] = {0.0, 0.0, 0.0, 0.0};
    bool odd = false;
    for (int64_t c = (int64_t)blockIdx.x * kBlock + threadIdx.x; c < a.n; c += (int64_t)gridDim.x * kBlock) {
        if (a.flags[c] != kFluid) continue;
        Cells<SA, 1> qa;
        Cells<SB, 1> qb;
        qa.load(a, c);
        qb.load(b, c);
        cnt++;
        uint64_t mass;
        typename CellFix<RA>::J ja[3];
        typename CellFix<RB>::J jb[3];
        const bool oka = CellFix<RA>::of(qa.f[0], mass, ja), okb = CellFix<RB>::of(qb.f[0], mass, jb);
        if (oka && okb) {
            u128 e2 = 0, r2 = 0;
            for (int k = 0; k < 3; k++) {
                int64_t x = (int64_t)ja[k] << (61 - CellFix<RA>::kLsb), y = (int64_t)jb[k] << (61 - CellFix<RB>::kLsb);
                if (la) x = -x;
                if (lb) y = -y;
                e2 += square(x - y);
                r2 += square(y);
            }
            mx = (i128)e2 > mx ? (i128)e2 : mx;
            mr = (i128)r2 > mr ? (i128)r2 : mr;
            se.add(e2);
            sr.add(r2);
        } else {
            odd = true;
            double r, ua[3], ub[3];
            moments_double<RA>(qa.f[0], r, ua);
            moments_double<RB>(qb.f[0], r, ub);
            double e2 = 0.0, r2 = 0.0;
            for (int k = 0; k < 3; k++) {
                const double x = la ? -ua[k] : ua[k], y = lb ? -ub[k] : ub[k];
                e2 += (x - y) * (x - y);
                r2 += y * y;
            }
            dv[0] = fmax(dv[0], sqrt(e2));
            dv[1] += e2;
            dv[2] += r2;
            dv[3] = fmax(dv[3], sqrt(r2));
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    mx = warp_max(mx);
    se.hi = warp_sum(se.hi);
    sr.hi = warp_sum(sr.hi);
    se.lo = warp_sum(se.lo);
    sr.lo = warp_sum(sr.lo);
    mr = warp_max(mr);
    const i128 n = warp_sum((i128)cnt);
    if (lane == 0) {
        wred[warp][0] = mx; wred[warp][1] = se.hi; wred[warp][2] = sr.hi; wred[warp][3] = mr; wred[warp][4] = n;
        wlow[warp][0] = se.lo; wlow[warp][1] = sr.lo;
    }
    if (__syncthreads_or(odd)) {
        for (int k = 0; k < 4; k++) sh[k][threadIdx.x] = dv[k];
        __syncthreads();
        for (int w = kBlock / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w)
                for (int k = 0; k < 4; k++) {
                    const double v = sh[k][threadIdx.x + w];
                    if (k == 0 || k == 3) sh[k][threadIdx.x] = fmax(sh[k][threadIdx.x], v);
                    else sh[k][threadIdx.x] += v;
                }
            __syncthreads();
        }
    } else if (threadIdx.x < 4) {
        sh[threadIdx.x][0] = 0.0;
    }
    if (threadIdx.x < 5) {
        i128 v = wred[0][threadIdx.x];
        for (int w = 1; w < kBlock / 32; w++) {
            const i128 o = wred[w][threadIdx.x];
            if (threadIdx.x == 0 || threadIdx.x == 3) v = o > v ? o : v;
            else v += o;
        }
        CmpPartial &p = partial[blockIdx.x];
        if (threadIdx.x < 4) {
            p.fix[threadIdx.x] = v;
            p.acc[threadIdx.x] = sh[threadIdx.x][0];
        } else {
            p.cells = (double)(int64_t)v;
        }
    } else if (threadIdx.x < 7) {
        const int k = threadIdx.x - 5;
        uint64_t v = 0;
        for (int w = 0; w < kBlock / 32; w++) v += wlow[w][k];
        partial[blockIdx.x].low[k] = v;
    }
}

__global__ void __launch_bounds__(160) k_compare_final(const CmpPartial *partial, int nblocks, double *out) {
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool is_max = q == 0 || q == 3;
    i128 v = 0;
    uint64_t low = 0;
    double a = 0.0;
    for (int b = lane; b < nblocks; b += 32) {
        if (q == 1 || q == 2) low += partial[b].low[q - 1];
        const i128 o = q < 4 ? partial[b].fix[q] : (i128)0;
        const double s = q < 4 ? partial[b].acc[q] : partial[b].cells;
        if (is_max) {
            v = o > v ? o : v;
            a = fmax(a, s);
        } else {
            v += o;
            a += s;
        }
    }
    v = is_max ? warp_max(v) : warp_sum(v);
    low = warp_sum(low);
    v += (i128)(low >> 32);
    for (int o = 16; o > 0; o >>= 1) {
        const double s = __shfl_down_sync(0xffffffffu, a, o);
        if (lane + o < 32) a = is_max ? fmax(a, s) : a + s;
    }
    if (lane == 0) out[q] = is_max ? fmax(a, sqrt(to_double(v, 122))) : a + to_double(v, 90, (uint32_t)low);
}

int red_blocks(const LatDesc &d, int per_thread) {
    return (int)std::min<int64_t>(std::min(kRedBlocks, 4 * sm_count()),
                                  std::max<int64_t>(1, grid_for((d.n + per_thread - 1) / per_thread)));
}

template <typename S>
int reduce_t(const LatDesc &d, int layout, RedPartial *partial, double *res, cudaStream_t st) {
    using F = CellFix<typename Store<S>::R>;
    const int blocks = red_blocks(d, sizeof(typename Store<S>::R) == 4 ? 2 : 1);
    k_reduce<S><<<blocks, kBlock, 0, st>>>(d, layout & 1, partial);
    CU(cudaGetLastError());
    k_reduce_final<<<1, 160, 0, st>>>(partial, blocks, F::kLsb, F::kLsb == 31 ? 62 : 90, res);
    CU(cudaGetLastError());
    return 0;
}

int reduce(const lbm_lattice *l, int layout, void *work, double out[5], cudaStream_t st) {
    RedPartial *partial = (RedPartial *)work;
    double *res = (double *)(partial + kRedBlocks);
    int rc = 0;
    switch (l->storage) {
        case kF32: rc = reduce_t<float>(l->h, layout, partial, res, st); break;
        case kF64: rc = reduce_t<double>(l->h, layout, partial, res, st); break;
        case kF16: rc = reduce_t<__half>(l->h, layout, partial, res, st); break;
        case kBF16: rc = reduce_t<__nv_bfloat16>(l->h, layout, partial, res, st); break;
        case kC16: rc = reduce_t<c16_t>(l->h, layout, partial, res, st); break;
    }
    if (rc) return rc;
    CU(cudaMemcpyAsync(out, res, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    return 0;
}

constexpr size_t kRedBytes = kRedBlocks * sizeof(RedPartial) + 8 * sizeof(double);

// Some callers must not allocate device memory: a serving loop that has
// handed every free byte of HBM to resident fields under a budget, a monitor
// thread that checks conservation while other streams run and cannot take
// the device-wide synchronisation cudaMalloc/cudaFree may imply, or a host
// framework whose own allocator owns the device.  For them the partial sums
// of the conservation reduction live in this fixed array instead of the
// lattice's staging buffer.  The array exists once per GPU that loads this
// library and stays allocated until the process exits.  Every call reuses it:
// each call writes every partial it later reads, so nothing has to be
// cleared, but two calls whose work overlaps on the GPU (different streams,
// no ordering) race on it.
constexpr int64_t kNoallocCells = 134217728;  // 512^3
static __device__ __align__(256) unsigned char g_reduce_scratch[kRedBytes];

// Device address of g_reduce_scratch, looked up once per device with that
// device current (the host-side symbol is not a device address).
int static_scratch(void **out) {
    static std::mutex mu;
    static void *addr[128] = {};
    int dev = 0;
    CU(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) return fail("device ordinal out of range");
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        CU(cudaGetSymbolAddress(&p, g_reduce_scratch));
        addr[dev] = p;
    }
    *out = addr[dev];
    return 0;
}
}  // namespace

extern "C" {

int lbm_cu_reduce_conserved(lbm_lattice *l, int layout, double out[5], void *stream) {
    if (!l || !out) return fail("NULL argument");
    if (ensure_stage(l, kRedBytes)) return -1;
    return reduce(l, layout, l->stage, out, S(stream));
}

int lbm_cu_reduce_conserved_noalloc(lbm_lattice *l, int layout, double out[5], void *stream) {
    if (!l || !out) return fail("NULL argument");
    if (l->n > kNoallocCells)
        return fail("lattice has " + std::to_string(l->n) + " cells; the no-allocation reduction handles at most " +
                    std::to_string(kNoallocCells));
    void *work = nullptr;
    if (static_scratch(&work)) return -1;
    return reduce(l, layout, work, out, S(stream));
}

int lbm_cu_compare_velocity(lbm_lattice *a, int layout_a, lbm_lattice *b, int layout_b, double out[5],
                            void *stream) {
    if (!a || !b || !out) return fail("NULL argument");
    if (a->nx != b->nx || a->ny != b->ny || a->nz != b->nz) return fail("lattices differ in size");
    if (ensure_stage(a, kRedBytes)) return -1;
    CmpPartial *partial = (CmpPartial *)a->stage;
    double *res = (double *)((RedPartial *)a->stage + kRedBlocks);
    const int blocks = red_blocks(a->h, 1);
    cudaStream_t st = S(stream);
#define CMP(SA_, SB_) k_compare<SA_, SB_><<<blocks, kBlock, 0, st>>>(a->h, layout_a & 1, b->h, layout_b & 1, partial)
#define CMPB(SA_)                                   \
    switch (b->storage) {                           \
        case kF32: CMP(SA_, float); break;          \
        case kF64: CMP(SA_, double); break;         \
        case kF16: CMP(SA_, __half); break;         \
        case kBF16: CMP(SA_, __nv_bfloat16); break; \
        case kC16: CMP(SA_, c16_t); break;          \
    }
    switch (a->storage) {
        case kF32: CMPB(float); break;
        case kF64: CMPB(double); break;
        case kF16: CMPB(__half); break;
        case kBF16: CMPB(__nv_bfloat16); break;
        case kC16: CMPB(c16_t); break;
    }
#undef CMPB
#undef CMP
    CU(cudaGetLastError());
    k_compare_final<<<1, 160, 0, st>>>(partial, blocks, res);
    CU(cudaGetLastError());
    CU(cudaMemcpyAsync(out, res, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    return 0;
}

}  // extern "C"
