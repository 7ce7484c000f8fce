// Host check of the table-driven cosine (pagmo2_gb300/csrc/trig_table.h) next
// to whole, half and quarter turns: 2^62 exactly at a whole turn, never more,
// never less than -2^62, and rastrigin rows of zeros and of small elements
// (whose exact value is not negative) never below 0. Prints "<values> <rows>
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
    std::mt19937_64 g(20261206);
    long values = 0, rows = 0, violations = 0;
    const auto see = [&](uint64_t f) {
        int64_t s, c;
        sincos(f, tab.data(), s, c);
        if (c > one || c < -one) ++violations;
        ++values;
    };
    for (uint64_t q = 0; q < 4; ++q) {
        const uint64_t at = q << 62;
        for (uint64_t d = 0; d <= 200000; ++d) {
            see(at + d);
            see(at - d);
        }
        for (int i = 0; i < 400000; ++i) {
            const uint64_t d = g() >> (12 + g() % 50);
            see(at + d);
            see(at - d);
        }
    }
    int64_t s, c;
    sincos(0u, tab.data(), s, c);
    if (c != one) ++violations;
    const auto row = [&](uint64_t n, double x) {
        sum96 sq{0u, 0}, cs{0u, 0};
        for (uint64_t i = 0; i < n; ++i) {
            add(sq, square_q52(magnitude_q58(x)));
            add(cs, cos_of(reduce(turn_of_periods(x), tab.data())));
        }
        ++rows;
        return rastrigin_value(sq, cs, n);
    };
    for (uint64_t n : {1u, 2u, 50u, 1000u, 4097u}) {
        if (row(n, 0.0) != 0.0 || row(n, -0.0) != 0.0 || row(n, 1e-310) != 0.0) ++violations;
        for (int i = 0; i < 200; ++i) {
            const double x = std::ldexp(1.0 + static_cast<double>(g() >> 11) * 0x1p-53, -static_cast<int>(g() % 70));
            if (!(row(n, x) >= 0.0)) ++violations;
        }
    }
    std::printf("%ld %ld %ld\n", values, rows, violations);
    return violations == 0 ? 0 : 1;
}
