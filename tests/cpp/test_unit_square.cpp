// Host check of DTLZ's squares (x - 1/2)^2 on [0, 1] in Q62
// (pagmo2_gb300/csrc/trig_table.h) against long double: within 0.75 units (the
// rounding and the low word's square), x's bits below 2^-62 beside them; 0 at
// 1/2, 2^60 at 0 and 1, and a mean error below 0.01 units. Prints "<values>
// <worst> <mean> <violations>"; exit 1 on a violation.
#include "trig_table.h"

#include <cmath>
#include <cstdio>
#include <random>

int main()
{
    using namespace pgx::trigtab;
    std::mt19937_64 g(20261211);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    long values = 0, violations = 0;
    long double worst = 0, sum = 0;
    if (centred_square_q62(unit_q62(0.5)) != 0) ++violations;
    for (double x : {0.0, 1.0, 5e-324, 1e-300})
        if (centred_square_q62(unit_q62(x)) != int64_t{1} << 60) ++violations;
    for (int i = 0; i < 400000; ++i) {
        double x = (i & 1) ? U(g) : 0.5 + std::ldexp(U(g) - 0.5, -static_cast<int>(g() % 50));
        if (i < 2000) x = std::ldexp(U(g), -static_cast<int>(g() % 30)); // next to 0
        else if (i < 4000) x = 1.0 - std::ldexp(U(g), -static_cast<int>(g() % 50));
        if (!in_unit(x)) continue;
        const long double d = static_cast<long double>(x) - 0.5L;
        const long double err = static_cast<long double>(centred_square_q62(unit_q62(x))) - std::ldexp(d * d, 62);
        if (!(std::fabs(err) <= 0.75L + (x < 0x1p-9 ? 1.0L : 0.0L) + std::ldexp(d * d, -2))) ++violations; // (long double's own rounding last)
        if (std::fabs(err) > worst) worst = std::fabs(err);
        sum += err;
        ++values;
    }
    const long double mean = sum / values;
    if (!(std::fabs(mean) <= 0.01L)) ++violations;
    std::printf("%ld %.3Lf %.4Lf %ld\n", values, worst, mean, violations);
    return violations == 0 ? 0 : 1;
}
