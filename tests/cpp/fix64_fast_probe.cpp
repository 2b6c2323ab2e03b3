// The integer collision of double populations in fast flows, up to the speeds
// that fx_flow accepts: accepted there, bit for bit the double arithmetic, and
// without intermediate roundings closer to long double than it.
// Usage: fix64_fast_probe SEED COUNT; exit status 1 and a line per mismatch.
#define main fix64_probe_main
#include "fix64_probe.cpp"
#undef main

int main(int argc, char **argv) {
    std::mt19937_64 g(argc > 1 ? atoi(argv[1]) : 1);
    const long count = argc > 2 ? atol(argv[2]) : 100000;
    const auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    long used = 0, refused = 0, outside = 0, bad = 0;
    double sum_grid = 0, sum_double = 0, max_grid = 0, max_double = 0;
    for (long n = 0; n < count; n++) {
        // speeds on both sides of the bound: two components that add up to 0.25 (1 +- e), a third below either
        const double e = n % 4 ? std::pow(10.0, U(-9, -0.3)) : 0.0, part = n % 3 ? U(0, 1) : 1.0;
        double v[3];
        const int a = (int)(g() % 3), b = (a + 1 + (int)(g() % 2)) % 3, c = 3 - a - b;
        v[a] = 0.25 * part * (1 - e * (n % 5 ? 1 : -1));
        v[b] = 0.25 * (1 - part) * (1 - e);
        v[c] = U(0, 1) * std::min(v[a], v[b]);
        for (double &x : v)
            if (g() & 1) x = -x;
        const double r = n % 7 ? U(0.95, 1.05) : U(0.875, 1.1), u2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
        double f[19], m[4], o[19], dp, w[3];
        equilibria<double>(v[0], v[1], v[2], r - 1.5 * u2, f);
        if (n % 2)
            for (int i = 0; i < 19; i++) f[i] *= 1 + std::pow(10.0, U(-12, -2)) * U(-1, 1);
        if (!fx_ordinary(f)) continue;
        const bool beta = g() & 1;
        Fx x[19], mx[4];
        for (int i = 0; i < 19; i++) x[i] = fx_of(f[i]);
        moments(x, beta, mx);
        moments(f, beta, m);
        const double s[3] = {std::fabs(m[1]), std::fabs(m[2]), std::fabs(m[3])};
        const double two = s[0] + s[1] + s[2] - std::min(s[0], std::min(s[1], s[2]));
        if (!fx_flow(mx[0], mx[1], mx[2], mx[3])) {
            refused++;
            if (two < 0.25 - 0x1p-27 && m[0] > 0.875 && m[0] < 1.875 && bad++ < 10)
                printf("refused: %g %g %g, density %g\n", m[1], m[2], m[3], m[0]);
            continue;
        }
        outside += two > 0.25;
        used++;
        const double tau0 = U(0.5005, 1.5), les = g() % 4 ? U(0, 5) : 0.0;
        long double fl[19], ml[4];
        for (int i = 0; i < 19; i++) fl[i] = f[i];
        if (les != 0) fx_collide<true>(x, mx[0], mx[1], mx[2], mx[3], 1 / tau0, tau0, les, o, dp, w[0], w[1], w[2]);
        else fx_collide<false>(x, mx[0], mx[1], mx[2], mx[3], 1 / tau0, tau0, les, o, dp, w[0], w[1], w[2]);
        const double want = collide<double>(f, m, 1 / tau0, tau0, les);
        if (bits_of(dp) != bits_of(want) && bad++ < 10) printf("dd_param %a instead of %a\n", dp, want);
        for (int i = 0; i < 19; i++)
            if (bits_of(o[i]) != bits_of(f[i]) && bad++ < 10) printf("population %d: %a instead of %a\n", i, o[i], f[i]);
        moments(fl, beta, ml);
        collide<long double>(fl, ml, 1 / tau0, tau0, les);
        double rho, q;
        const bool ok = les != 0 ? fq_collide<true>(x, 1 / tau0, tau0, les, true, o, rho, q, w[0], w[1], w[2])
                                 : fq_collide<false>(x, 1 / tau0, tau0, les, true, o, rho, q, w[0], w[1], w[2]);
        if (!ok) continue;
        for (int i = 0; i < 19; i++) {
            if (fl[i] < 0x1p-10L) continue;
            const double eo = (double)((o[i] - fl[i]) / fl[i]), ef = (double)((f[i] - fl[i]) / fl[i]);
            sum_grid += eo * eo;
            sum_double += ef * ef;
            max_grid = std::max(max_grid, std::fabs(eo));
            max_double = std::max(max_double, std::fabs(ef));
        }
    }
    printf("%ld cells used, %ld refused, %ld beyond the bound, %ld mismatches\n", used, refused, outside, bad);
    printf("without roundings: mean square %.3g (double %.3g), largest %.3g (%.3g)\n", sum_grid, sum_double, max_grid,
           max_double);
    return bad || used < count / 4 || !refused || !(sum_grid < sum_double) || !(max_grid < max_double);
}
