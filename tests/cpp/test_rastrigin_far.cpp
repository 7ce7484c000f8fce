// Host check of rastrigin's squares for 8 <= |x| < 2^11 (pagmo2_gb300/csrc/trig_table.h):
// against the exact 106-bit square, the floor of its high 64 bits and one more
// below 2^5 (1 unit of Q52 there, 2^(2 e - 10) from 2^5 on), and sums over the
// whole range with usual elements. Prints "<values> <worst, units of that>
// <violations>"; exit 1 on a violation.
#include "trig_table.h"

#include <cmath>
#include <cstdio>
#include <random>

int main()
{
    using namespace pgx::trigtab;
    std::mt19937_64 g(20261209);
    std::uniform_real_distribution<double> U(0.5, 1.0);
    long values = 0, violations = 0;
    double worst = 0;
    const auto number = [](const sum96 &a) { return (static_cast<__int128>(a.hi) << 64) + static_cast<__int128>(a.lo); };
    for (int e = 4; e <= 11; ++e)
        for (int i = 0; i < 100000; ++i) {
            double x = std::ldexp(i == 0 ? 0.5 : (i == 1 ? std::nextafter(1.0, 0.0) : U(g)), e);
            if (i & 1) x = -x;
            if (exponent_bits(x) >= rastrigin_end(50)) ++violations;
            // x = m 2^p: x^2 2^52 = m^2 2^(2 p + 52)
            const int p = static_cast<int>(exponent_bits(x)) - 1075;
            const unsigned __int128 m2 = static_cast<unsigned __int128>(mantissa_of(x)) * mantissa_of(x);
            const int down = -(2 * p + 52);
            const __int128 want = static_cast<__int128>(m2 >> down);
            const int k = 2 * (e - 1) - 10;
            const double err = static_cast<double>(want - number(square_far(x))) / std::ldexp(1.0, k > 0 ? k : 0);
            if (!(err >= 0 && err <= 1.0)) ++violations;
            if (err > worst) worst = err;
            ++values;
        }
    if (rastrigin_end(1u << 20) != 1034u || rastrigin_end((1u << 20) + 1u) != 1026u) ++violations;
    // the most that fits: 2^20 of the largest
    sum96 s{0u, 0};
    const double top = std::nextafter(2048.0, 0.0);
    for (uint32_t i = 0; i < (1u << 20); ++i) add(s, square_far(top));
    if (number(s) != number(square_far(top)) << 20 || s.hi < 0) ++violations;
    const double f = rastrigin_value(s, sum96{0u, static_cast<int32_t>(1 << 18)}, 1u << 20); // 2^20 cosines of 1
    if (std::fabs(f / std::ldexp(top * top, 20) - 1.0) > 1e-15) ++violations;
    std::printf("%ld %.3f %ld\n", values, worst, violations);
    return violations == 0 ? 0 : 1;
}
