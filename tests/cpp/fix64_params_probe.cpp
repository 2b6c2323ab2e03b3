// The integer collision of double populations under relaxation parameters
// outside the ordinary ones (infinite, not a number, negative, huge, tiny):
// they are either refused (fx_params) or give the bits of the double
// arithmetic, up to the ends of what is accepted.
// Usage: fix64_params_probe COUNT; exit status 1 and a line per mismatch.
#define main fix64_probe_main
#include "fix64_probe.cpp"
#undef main

static bool same(double a, double b) { return (a != a && b != b) || bits_of(a) == bits_of(b); }

int main(int argc, char **argv) {
    const long count = argc > 1 ? atol(argv[1]) : 1000;
    const double inf = INFINITY, nan = NAN;
    struct P {
        double inv_tau, tau0, les;
        bool ordinary;  // has to be accepted
    };
    const P params[] = {{1.9, 1 / 1.9, 0, true},  {0.0, 0, 0, true},         {-1.5, 0, 0, true},      {1e308, 0, 0, true},
                        {1e-310, 0, 0, true},     {inf, 0, 0, false},        {-inf, 0, 0, false},     {nan, 0, 0, false},
                        {1.9, 0.53, 0.7, true},   {1.9, 0.53, 1e-300, true}, {1.9, 1e10, 0.7, true},  {1.9, 1e30, 0.7, false},
                        {1.9, 1e155, 0.7, false}, {1.9, 1e300, 0.7, false},  {1.9, inf, 0.7, false},  {1.9, 0.53, -0.01, false},
                        {1.9, 0.53, -1, false},   {1.9, 0.53, -1e6, false},  {1.9, 0.53, 1e29, true}, {1.9, 0.53, 1e300, false},
                        {1.9, 0x1p50, 0x1p100, true}, {1.9, 0.5, 0x1p100, true}, {1.9, 0x1p50, 1e-300, true},
                        {1.9, 0.53, inf, false},  {1.9, 0.53, -inf, false},  {1.9, 0.53, nan, false}};
    std::mt19937_64 g(5);
    const auto U = [&](double a, double b) { return a + (b - a) * ((g() >> 11) * 0x1p-53); };
    long bad = 0;
    double rest[19];
    equilibria<double>(0, 0, 0, 1.0, rest);
    for (const P &p : params) {
        if (!fx_params(p.inv_tau, p.tau0, p.les)) {
            if (p.ordinary && ++bad) printf("inv_tau %g tau0 %g les %g refused\n", p.inv_tau, p.tau0, p.les);
            continue;
        }
        for (long n = 0; n < count; n++) {
            double f[19], o[19], m[4], v[3], dp = 0;
            const double amp = n ? std::pow(10.0, U(-15, -0.6)) : 0.0;
            for (int i = 0; i < 19; i++) f[i] = rest[i] * (1 + amp * U(-1, 1));
            if (!fx_ordinary(f)) continue;
            Fx x[19], mx[4];
            for (int i = 0; i < 19; i++) x[i] = fx_of(f[i]);
            moments(x, n & 1, mx);
            moments(f, n & 1, m);
            if (!fx_flow(mx[0], mx[1], mx[2], mx[3])) continue;
            if (p.les != 0)
                fx_collide<true>(x, mx[0], mx[1], mx[2], mx[3], p.inv_tau, p.tau0, p.les, o, dp, v[0], v[1], v[2]);
            else
                fx_collide<false>(x, mx[0], mx[1], mx[2], mx[3], p.inv_tau, p.tau0, p.les, o, dp, v[0], v[1], v[2]);
            collide<double>(f, m, p.inv_tau, p.tau0, p.les);
            for (int i = 0; i < 19; i++)
                if (!same(o[i], f[i]) && bad++ < 20)
                    printf("inv_tau %g tau0 %g les %g: %a instead of %a\n", p.inv_tau, p.tau0, p.les, o[i], f[i]);
        }
    }
    printf("%ld mismatches\n", bad);
    return bad != 0;
}
