// Host check of fx_state (fx_tables.h): the last state whose spot is not above a level, against extended
// precision, for the barriers, spots and ranges that the FP64 Dupire kernel takes.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#include "fx_tables.h"

typedef long double real;  // 64 or more bits on both build hosts

int main()
{
    std::mt19937_64 g(4);
    std::uniform_real_distribution<double> un(0.0, 1.0);
    long bad = 0, n = 0;
    real worst = 0.0L;
    auto check = [&](double spot, double level, int r) {
        const double x0 = std::log(spot);
        // in units of the state; the extended logarithm is good to 2^-63 of it (at most 2^-59 for |log| < 16)
        const real ref = ldexpl(logl((real)level) - (real)x0, cf::FX_Y - r), own = ldexpl(16.0L, cf::FX_Y - r - 63);
        const long long y = cf::fx_state(level, x0, r);
        const real below = ref - (real)y;  // in [0, 1)
        if (!(below >= -own && below < 1.0L + own)) ++bad;
        worst = std::max(worst, fabsl(below - 0.5L));
        ++n;
    };
    for (int r = 0; r <= 4; ++r)
    {
        for (int i = 0; i < 20000; ++i)
        {
            const double spot = std::exp(-6.0 + 18.0 * un(g)), level = spot * std::exp(0.6 * un(g) - 0.1);
            check(spot, level, r);
        }
        for (double s : {1.0, 1.5, 90.0, 100.0, 110.0, 1e-3, 1e5})
            for (double b : {1.0, 1.0 + 1e-12, 1.2, 1.49, 1.5, 1.51, 3.0, 0.5}) check(s, s * b, r);
        const bool ends = cf::fx_state(0.0, 4.6, r) == INT64_MIN && cf::fx_state(-5.0, 4.6, r) == INT64_MIN &&
                          cf::fx_state((double)INFINITY, 4.6, r) == INT64_MAX && cf::fx_state(1e300, 4.6, 0) == INT64_MAX &&
                          cf::fx_state(1e-300, 4.6, 0) == INT64_MIN && cf::fx_state(1.0, 0.0, r) == 0;
        if (!ends) ++bad;
    }
    std::printf("%s %ld levels, worst %.2Lg units from the middle of their state\n", bad ? "BAD" : "ok", n, worst);
    return bad != 0;
}
