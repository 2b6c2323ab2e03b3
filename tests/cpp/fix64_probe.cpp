// Compares the integer collision of double populations (lbm_fix64.cuh) with
// the same operations in double arithmetic, bit for bit, on random cells, and
// its square root and reciprocal with the correctly rounded ones; and the
// collision without intermediate roundings with long double arithmetic: its
// errors have to be smaller than those of double arithmetic.
// Usage: fix64_probe SEED COUNT; exit status 1 and a line per mismatch.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "lbm_fix64.cuh"

using namespace lbm;

static const int kOrderBeta[19] = {3, 2, 0, 1, 4, 5, 6, 7, 8, 9, 10, 11, 13, 12, 15, 14, 17, 16, 18};
static const int kDir[3][19] = {{1, -1, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1, 0, 0, 0, 0, 0, 0, 0},
                                {0, 0, 1, -1, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 0},
                                {0, 0, 0, 0, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1, 1, -1, 0}};
static const double c18 = (double)(1.0f / 18.0f), c36 = (double)(1.0f / 36.0f), c3 = (double)(1.0f / 3.0f);

// Sequential sums in the order of a beta or an alpha step.
template <typename M> void moments(const M f[19], bool beta, M out[4]) {
    bool set[4] = {false, false, false, false};
    for (int n = 0; n < 19; n++) {
        const int i = beta ? kOrderBeta[n] : n;
        for (int q = 0; q < 4; q++) {
            const int e = q == 0 ? 1 : kDir[q - 1][i];
            if (!e) continue;
            if (!set[q]) out[q] = e > 0 ? f[i] : -f[i];
            else if (e > 0) out[q] += f[i];
            else out[q] -= f[i];
            set[q] = true;
        }
    }
}
template <typename T> static void equilibria(T vx, T vy, T vz, T r, T e[19]) {
    const T s[9] = {vx, vy, vx + vy, vx - vy, vx + vz, vx - vz, vy + vz, vy - vz, vz};
    for (int k = 0; k < 9; k++) {
        const T c = k < 2 || k == 8 ? c18 : c36, s2 = s[k] * s[k];
        e[2 * k] = c * ((r + T(3) * s[k]) + T(4.5) * s2);
        e[2 * k + 1] = c * ((r + T(-3) * s[k]) + T(4.5) * s2);
    }
    e[18] = T(c3) * r;
}
template <typename T> static T collide(T f[19], const T m[4], T inv_tau, T tau0, T les) {
    const T r = m[0], vx = m[1], vy = m[2], vz = m[3];
    const T dp = r - T(1.5) * ((vx * vx + vy * vy) + vz * vz);
    T w = inv_tau;
    if (les != 0) {
        T p[9];
        for (int k = 0; k < 9; k++) p[k] = f[2 * k] + f[2 * k + 1];
        const T r3 = r * T(c3);
        const T a = (((((p[0] + p[2]) + p[3]) + p[4]) + p[5]) - r3) - vx * vx;
        const T b = (((((p[1] + p[2]) + p[3]) + p[6]) + p[7]) - r3) - vy * vy;
        const T c = (((((p[4] + p[5]) + p[6]) + p[7]) + p[8]) - r3) - vz * vz;
        const T d = (p[2] - p[3]) - vx * vy, e = (p[4] - p[5]) - vx * vz, g = (p[6] - p[7]) - vy * vz;
        const T q = ((a * a + b * b) + c * c) + T(2) * ((d * d + e * e) + g * g);
        w = T(1) / (T(0.5) * (tau0 + std::sqrt(tau0 * tau0 + les * std::sqrt(q))));
    }
    T e[19];
    equilibria(vx, vy, vz, dp, e);
    for (int i = 0; i < 19; i++) f[i] += w * (e[i] - f[i]);
    return dp;
}

int main(int argc, char **argv) {
    std::mt19937_64 g(argc > 1 ? atoi(argv[1]) : 1);
    const long count = argc > 2 ? atol(argv[2]) : 100000;
    const auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    long used = 0, bad = 0;
    double sum_grid = 0, sum_double = 0, max_grid = 0, max_double = 0;  // errors against long double
    const auto differ = [&](const char *what, double got, double want) {
        if (bits_of(got) == bits_of(want)) return;
        if (bad++ < 10) printf("%s: %a instead of %a\n", what, got, want);
    };
    double rest[19];
    equilibria<double>(0, 0, 0, 1.0, rest);
    for (long n = 0; n < count; n++) {
        double f[19];
        const int mode = (int)(g() % 6);
        const double amp = std::pow(10.0, U(-12, -0.3));
        if (mode == 0 || mode == 5) {  // noise around rest, some of it in few bits or symmetric
            for (int i = 0; i < 19; i++) f[i] = rest[i] * (1 + amp * U(-1, 1));
            if (mode == 5)
                for (int i = 0; i < 19; i++) {
                    if (g() % 3 == 0) f[i] = (float)f[i];
                    if ((i & 1) && g() % 3 == 0) f[i] = f[i - 1];
                }
        } else if (mode < 4) {  // equilibria of flows up to and beyond the accepted speed
            const double u = mode == 1 ? 0.13 : mode == 2 ? 0.02 : 1e-5, r = g() % 4 ? U(0.87, 1.3) : 1.0;
            double v[3] = {U(-u, u), U(-u, u), U(-u, u)};
            for (int a = 0; a < 3; a++)
                if (g() % 8 == 0) v[a] = a ? v[0] : 0.0;
            equilibria<double>(v[0], v[1], v[2], r - 1.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]), f);
            if (g() % 3)
                for (int i = 0; i < 19; i++) f[i] *= 1 + 0.1 * amp * U(-1, 1);
        } else {  // anything, out of range too
            for (int i = 0; i < 18; i++) f[i] = std::exp2(U(-9.1, -2.95));
            f[18] = U(0.2, 0.5);
        }
        if (!fx_ordinary(f)) continue;
        const bool beta = g() & 1;
        const double tau0 = U(0.5005, 1.5), les = g() % 4 ? U(0, 5) : 0.0;
        Fx x[19], mx[4];
        for (int i = 0; i < 19; i++) x[i] = fx_of(f[i]);
        double m[4], o[19], dp, v[3];
        long double fl[19], ml[4];
        for (int i = 0; i < 19; i++) fl[i] = f[i];
        moments(x, beta, mx);
        moments(f, beta, m);
        differ("density", fx_pos(mx[0]), m[0]);
        for (int a = 1; a < 4; a++) differ("momentum", fx_double(mx[a]), m[a]);
        if (!fx_flow(mx[0], mx[1], mx[2], mx[3])) continue;
        used++;
        if (les != 0) fx_collide<true>(x, mx[0], mx[1], mx[2], mx[3], 1 / tau0, tau0, les, o, dp, v[0], v[1], v[2]);
        else fx_collide<false>(x, mx[0], mx[1], mx[2], mx[3], 1 / tau0, tau0, les, o, dp, v[0], v[1], v[2]);
        differ("dd_param", dp, collide<double>(f, m, 1 / tau0, tau0, les));
        for (int i = 0; i < 19; i++) differ("population", o[i], f[i]);
        moments(fl, beta, ml);
        collide<long double>(fl, ml, 1 / tau0, tau0, les);
        double rho, a;
        const bool ok = les != 0 ? fq_collide<true>(x, 1 / tau0, tau0, les, true, o, rho, a, v[0], v[1], v[2])
                                 : fq_collide<false>(x, 1 / tau0, tau0, les, true, o, rho, a, v[0], v[1], v[2]);
        if (!ok) continue;
        for (int i = 0; i < 19; i++) {
            const double eo = (double)((o[i] - fl[i]) / fl[i]), ef = (double)((f[i] - fl[i]) / fl[i]);
            if (fl[i] < 0x1p-10L) continue;
            sum_grid += eo * eo;
            sum_double += ef * ef;
            max_grid = std::max(max_grid, std::fabs(eo));
            max_double = std::max(max_double, std::fabs(ef));
        }
    }
    for (long n = 0; n < count; n++) {
        double a = n % 3 ? std::exp2(U(-119.9, 99.9)) : std::exp2(U(-3, 3));
        if (n % 11 == 0) a = std::pow(std::floor(U(1, 67108864)), 2) * (n % 2 ? 1 : 2) + n % 2;
        differ("square root", sqrt_int(a), std::sqrt(a));
        double t = n % 5 ? U(0.3, 4) : std::exp2(U(-59, 59));
        if (n % 9 == 0) t = std::exp2(std::floor(U(-50, 50)));
        if (n % 10 == 0) t = 2 - 0x1p-52 * (double)(n % 1000 + 1);
        differ("reciprocal", rcp_int(t), 1.0 / t);
        double lid = n % 9 ? U(-0.13, 0.13) * (n % 5 ? 1 : 0.1) : 0.0;
        if (fx_lid_speed(lid)) {
            double o[19], e[19], dp;
            const double want = 1.0 - 1.5 * ((lid * lid + 0.0) + 0.0);
            fx_lid(lid, o, dp);
            equilibria<double>(lid, 0, 0, want, e);
            differ("lid dd_param", dp, want);
            for (int i = 0; i < 19; i++) differ("lid population", o[i], e[i]);
        }
    }
    printf("%ld cells used, %ld mismatches\n", used, bad);
    printf("without roundings: mean square %.3g (double %.3g), largest %.3g (%.3g)\n", sum_grid, sum_double, max_grid,
           max_double);
    return bad || used < count / 4 || !(sum_grid < sum_double) || !(max_grid < max_double);
}
