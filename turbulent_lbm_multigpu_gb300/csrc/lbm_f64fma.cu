// lbm_f64fma.cu -- the one-cell step kernels for double populations without
// the reference's intermediate roundings.
//
// Cells of ordinary flows are collided in 62-bit integers (fq_collide,
// lbm_fix64.cuh): exact sums, products cut at 2^-61, one rounding per
// population at the end.  Other cells run the double expressions, which this
// translation unit alone compiles with -fmad=true, so that the compiler may
// contract each product that feeds a sum into one FP64 fused multiply-add.
// Either way a step differs from the reference arithmetic by a few units in
// the last place (a relative 1e-15, well inside the 1e-12 per-step bound for
// double); against 128-bit arithmetic the integer form is off by 4e-17 RMS
// where fused double arithmetic is off by 2.3e-16.
//
// The kernels are instantiated for a storage tag type of their own (F64Fma:
// one double), so that their template instances can never be confused with
// the bit-exact k_beta<double> / k_alpha<double> of the other units.
#include "lbm_internal.h"

namespace lbm {
struct F64Fma {
    double v;
};
static_assert(sizeof(F64Fma) == sizeof(double), "same layout as double populations");

template <> struct Store<F64Fma> {
    using R = double;
    static constexpr int kDev = 0;
    __device__ static __forceinline__ R ld(const F64Fma *p, R) { return p->v; }
    __device__ static __forceinline__ void st(F64Fma *p, R v, R) { p->v = v; }
};
}  // namespace lbm

namespace lbm_rt {
int launch_step_f64_fma(int parity, bool les, const DomainArgs &a, int blocks, Dep dep, cudaStream_t st) {
    if (blocks <= 0) return 0;
    if (parity)
        return les ? launch_dep(dep, k_alpha<F64Fma, true>, blocks, kBlock, 0, st, a)
                   : launch_dep(dep, k_alpha<F64Fma, false>, blocks, kBlock, 0, st, a);
    return les ? launch_dep(dep, k_beta<F64Fma, true>, blocks, kBlock, 0, st, a)
               : launch_dep(dep, k_beta<F64Fma, false>, blocks, kBlock, 0, st, a);
}
}  // namespace lbm_rt
