// Host check of schwefel's elements outside 2^-20 <= |x| < 512
// (pagmo2_gb300/csrc/trig_table.h) against long double, in units of 2^-51: below
// 2^-20 within 1.5 (two floors, the sine's dropped term and the root), from 512
// to 2^14 within 2 2^k for |x| < 2^(9 + k) (the element's last place) and |x|
// (2^-57 + sqrt |x| 2^-58) (the sine's and its angle's). Signs, 0 and
// subnormals; sums of such terms. Prints "<values> <worst small> <worst large,
// of its bound> <violations>"; exit 1 on a violation.
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
    std::mt19937_64 g(20261208);
    std::uniform_real_distribution<double> U(0.5, 1.0);
    long values = 0, violations = 0;
    long double worst_s = 0, worst_l = 0;
    const auto number = [](const sum96 &a) {
        return std::ldexp(static_cast<long double>(a.hi), 64) + static_cast<long double>(a.lo);
    };
    const auto seed = [&](double x) { // one part in 2^21 off
        const long double v = std::ldexp(static_cast<long double>(sqrt_operand(x)), -62);
        const long double q32 = (1 + std::ldexp(2.0L * U(g) - 1.5L, -20)) / std::sqrt(v) * 4294967296.0L;
        return q32 >= 4294967295.0L ? 0xffffffffu : static_cast<uint32_t>(q32);
    };
    for (int e = -1080; e <= 14; e = e < -120 ? e + 20 : e + 1)
        for (int i = 0; i < 4000; ++i) {
            double x = std::ldexp(i == 0 ? 0.5 : (i == 1 ? std::nextafter(1.0, 0.0) : U(g)), e);
            if (i & 1) x = -x;
            if (schwefel_in_range(x) || !schwefel_far(x)) continue;
            const long double ax = std::fabs(static_cast<long double>(x)), root = std::sqrt(ax);
            const long double want = std::ldexp(static_cast<long double>(x) * std::sin(root), 51);
            const long double err = std::fabs(number(schwefel_far_term(x, seed(x), tab.data())) - want);
            if (e <= -20) {
                if (!(err <= 1.5L)) ++violations;
                if (err > worst_s) worst_s = err;
            } else {
                const long double bound = std::ldexp(2.0L, std::ilogb(x) - 8)
                                          + std::ldexp(ax * (std::ldexp(1.0L, -57) + std::ldexp(root, -58)), 51);
                if (!(err <= bound)) ++violations;
                if (err / bound > worst_l) worst_l = err / bound;
            }
            ++values;
        }
    for (double x : {0.0, -0.0, 5e-324, -1e-310, 1e-100})
        if (number(schwefel_far_term(x, seed(x), tab.data())) != 0) ++violations;
    sum96 s{0u, 0};
    long double want = 0;
    for (int i = 0; i < 100000; ++i) {
        const double x = 16383.0 * (2 * U(g) - 1) * ((g() & 1) ? 1 : -1);
        if (schwefel_in_range(x)) continue;
        const sum96 t = schwefel_far_term(x, seed(x), tab.data());
        add(s, t);
        want += number(t);
    }
    if (!(std::fabs(number(s) - want) <= std::fabs(want) * std::ldexp(1.0L, -40))) ++violations;
    std::printf("%ld %.3Lf %.3Lf %ld\n", values, worst_s, worst_l, violations);
    return violations == 0 ? 0 : 1;
}
