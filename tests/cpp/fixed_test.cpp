// Host check of fixed64.h: the integer split of a double into the accumulators' two words equals
// the floating form (rint at 2^-20, then at 2^-60) at every exponent it covers, ties included.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <random>

#include "fixed64.h"

static unsigned long long bits(double v)
{
    unsigned long long b;
    std::memcpy(&b, &v, 8);
    return b;
}

int main()
{
    std::mt19937_64 g(7);
    long bad = 0, n = 0;
    auto check = [&](double v) {
        long long hi = 0, lo = 0;
        const bool in = cf::fix_split_bits(bits(v), hi, lo);
        ++n;
        if (in != (std::fabs(v) < std::ldexp(1.0, 42)))
        {
            ++bad;
            return;
        }
        if (!in) return;
        const long long h = llrint(v * 1048576.0);
        const long long l = llrint((v - (double)h * (1.0 / 1048576.0)) * 1152921504606846976.0);
        if (((__int128)hi << 40) + lo != ((__int128)h << 40) + l) ++bad;
    };
    for (int e = -1074; e < 1024; ++e)
        for (int k = 0; k < 400; ++k)
        {
            // random mantissas, some cut to few bits so that halves of the unit occur
            unsigned long long m = g() & 0xfffffffffffffULL;
            if (k & 1) m &= ~0ULL << (g() % 52);
            const double v = std::ldexp(1.0 + std::ldexp((double)m, -52), e);
            check(v);
            check(-v);
        }
    for (const double v : std::initializer_list<double>{0.0, -0.0, (double)INFINITY, -(double)INFINITY, std::ldexp(1.0, 42), std::nextafter(std::ldexp(1.0, 42), 0.0),
                     std::ldexp(1.0, -61), std::ldexp(3.0, -61), std::ldexp(1.0, -62), 5e-324})
    {
        check(v);
        check(-v);
    }
    std::printf("%s split %ld values\n", bad ? "BAD" : "ok", n);
    return bad != 0;
}
