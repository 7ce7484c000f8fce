// Host check of griewank's factors for |x| < 2^-16 (pagmo2_gb300/csrc/trig_table.h)
// against long double: 1 - cos within 2 units of 2^-62 over all binades and
// columns, 0 for 0, subnormals and what rounds to 1, never negative; products
// of n such factors within n (2 + 1) units and never above 1. Prints "<values>
// <worst, units> <worst product, of its bound> <violations>"; exit 1 on a
// violation.
#include "trig_table.h"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

int main()
{
    using namespace pgx::trigtab;
    static const int64_t quarter[] = {PGX_TRIG_QUARTER_WAVE};
    std::vector<entry> tab(kN);
    for (uint32_t j = 0; j < kN; ++j) tab[j] = make_entry(quarter, j);
    std::mt19937_64 g(20261207);
    std::uniform_real_distribution<double> U(0.5, 1.0);
    long values = 0, violations = 0;
    long double worst = 0, worst_p = 0;
    const auto exact = [](double x, uint32_t i) { // (1 - cos) 2^62; the series' third term is below 2^-9 units
        const long double z = static_cast<long double>(x) * x / (i + 1.0L);
        return std::ldexp(z / 2 - z * z / 24, 62);
    };
    for (uint32_t i : {0u, 1u, 2u, 6u, 7u, 49u, 1023u, 1024u, 99999u}) {
        const column_factor c = make_column(i);
        for (int e = -1080; e <= -16; e = e < -60 ? e + 20 : e + 1)
            for (int q = 0; q < 2000; ++q) {
                double x = std::ldexp(q == 0 ? 0.5 : (q == 1 ? std::nextafter(1.0, 0.0) : U(g)), e);
                if (q & 1) x = -x;
                if (!griewank_small(x)) continue;
                const int32_t less = griewank_less(x, c, tab.data());
                const long double err = std::fabs(less - exact(x, i));
                if (less < 0 || !(err <= 2)) ++violations;
                if (err > worst) worst = err;
                ++values;
            }
        if (griewank_less(0.0, c, tab.data()) != 0 || griewank_less(-0.0, c, tab.data()) != 0
            || griewank_less(5e-324, c, tab.data()) != 0 || griewank_less(0x1p-40, c, tab.data()) != 0)
            ++violations;
    }
    const int64_t one = int64_t{1} << 62;
    for (int r = 0; r < 2000; ++r) {
        const uint32_t n = 1 + static_cast<uint32_t>(g() % 1000);
        const int e = -16 - static_cast<int>(g() % 20);
        int64_t p = one;
        long double want = 0; // log of the product
        for (uint32_t i = 0; i < n; ++i) {
            const double x = std::ldexp(U(g), e);
            p = scale_down(p, griewank_less(x, make_column(i), tab.data()));
            want += std::log1p(-std::ldexp(exact(x, i), -62));
        }
        const long double err = std::fabs(std::ldexp(static_cast<long double>(p - one), 0) - std::ldexp(std::expm1(want), 62)) / (3.0L * n);
        if (p > one || !(err <= 1)) ++violations;
        if (err > worst_p) worst_p = err;
        ++values;
    }
    std::printf("%ld %.3Lf %.3Lf %ld\n", values, worst, worst_p, violations);
    return violations == 0 ? 0 : 1;
}
