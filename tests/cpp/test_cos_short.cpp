// Host check of the short cosine (cos_short with reduce, pagmo2_gb300/csrc/trig_table.h):
// 2^62 exactly at a whole turn, never more, never less than -2^62, and within
// 2^-57 of long double over all steps of the table. Prints "<values> <worst>
// <violations>"; exit 1 on a violation.
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
    const int64_t one = int64_t{1} << 62;
    const long double pi = 3.141592653589793238462643383279502884L;
    std::mt19937_64 g(20261210);
    long values = 0, violations = 0;
    long double worst = 0;
    const auto see = [&](uint64_t f) {
        const int64_t c = cos_short(reduce(f, tab.data()));
        // the nearest quarter of a turn taken off exactly
        const uint64_t k = (f + (1ull << 61)) >> 62;
        const long double r = 2 * pi * std::ldexp(static_cast<long double>(static_cast<int64_t>(f - (k << 62))), -64);
        const long double want = (k & 1u) ? ((k & 2u) ? std::sin(r) : -std::sin(r)) : ((k & 2u) ? -std::cos(r) : std::cos(r));
        const long double err = std::fabs(std::ldexp(static_cast<long double>(c), -62) - want);
        if (c > one || c < -one || !(err <= std::ldexp(1.0L, -57))) ++violations;
        if (err > worst) worst = err;
        ++values;
    };
    for (uint64_t q = 0; q < 4; ++q)
        for (uint64_t d = 0; d <= 100000; ++d) {
            see((q << 62) + d);
            see((q << 62) - d);
            const uint64_t e = g() >> (12 + g() % 50);
            see((q << 62) + e);
            see((q << 62) - e);
        }
    for (uint64_t j = 0; j < 2 * kN; ++j)
        for (int i = 0; i < 500; ++i) see((j << (63 - kLogN)) + (g() >> (kLogN + 1)));
    if (cos_short(reduce(0u, tab.data())) != one) ++violations;
    std::printf("%ld %.3Le %ld\n", values, worst, violations);
    return violations == 0 ? 0 : 1;
}
