// Host check of the split of a double into the accumulators' two words (fixed64.h):
// * the low word of every accepted value is at most 2^39 in magnitude, the total is rint(v 2^60);
// * sums of many terms of one sign in two 64-bit words that wrap around: small and ordinary values,
//   equal and random ones;
// * the split of a node slab's 96-bit word, likewise.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "fixed64.h"

static unsigned long long bits(double v)
{
    unsigned long long b;
    std::memcpy(&b, &v, 8);
    return b;
}

static int words()
{
    std::mt19937_64 g(3);
    long bad = 0;
    auto check = [&](double v) {
        long long hi = 0, lo = 0;
        if (!cf::fix_split_bits(bits(v), hi, lo) || std::llabs(lo) > (1LL << 39)) ++bad;
        const double s = std::ldexp(std::fabs(v), 60);  // exact; below 2^102
        // rint of it: doubles of 2^53 or more are whole
        const __int128 t = s < 9007199254740992.0 ? (__int128)std::nearbyint(s) : (__int128)s;
        if (((__int128)hi << 40) + lo != (v < 0 ? -t : t)) ++bad;
    };
    for (int e = -70; e < 42; ++e)
        for (int k = 0; k < 2000; ++k)
        {
            unsigned long long m = g() & 0xfffffffffffffULL;
            if (k & 1) m &= ~0ULL << (g() % 52);
            if (k % 5 == 0) m = 0xfffffffffffffULL - g() % 3;
            const double v = std::ldexp(1.0 + std::ldexp((double)m, -52), e);
            check(v);
            check(-v);
        }
    std::printf("%s words\n", bad ? "BAD" : "ok");
    return bad != 0;
}

// n terms v(i) in wrapping 64-bit words, against the exact total.
template <class V>
static int sum(const char* what, long n, V&& v)
{
    unsigned long long H = 0, L = 0;
    __int128 exact = 0;
    for (long i = 0; i < n; ++i)
    {
        const double x = v(i);
        long long hi = 0, lo = 0;
        cf::fix_split_bits(bits(x), hi, lo);
        H += (unsigned long long)hi;
        L += (unsigned long long)lo;
        exact += (__int128)std::nearbyint(std::ldexp(x, 60));  // |x| < 2^-7, or few bits: below 2^53 or whole
    }
    const bool ok = ((__int128)(long long)H << 40) + (long long)L == exact;
    std::printf("%s %s\n", ok ? "ok" : "BAD", what);
    return !ok;
}

// Words of a node slab: the low part is at most 2^39, the total is the word; and the flushes of a run of
// 2^31 paths in sweeps of 128, each of a random positive total, stay in two 64-bit words.
static int slab()
{
    std::mt19937_64 g(8);
    long bad = 0;
    __int128 exact = 0;
    unsigned long long H = 0, L = 0;
    for (long i = 0; i < (3L << 23); ++i)
    {
        __int128 v = (__int128)(g() >> (i & 15));
        if (i & 1) v = (v << 20) ^ g();
        const bool neg = i >= (1L << 24) && (i & 2);
        if (neg) v = -v;
        long long hi, lo;
        cf::fix_split_slab((unsigned)v, (unsigned)(unsigned long long)(v >> 32), (unsigned)(unsigned long long)(v >> 64), hi, lo);
        if (lo < -(1LL << 39) || lo >= (1LL << 39) || ((__int128)hi << 40) + lo != v) ++bad;
        H += (unsigned long long)hi;
        L += (unsigned long long)lo;
        exact += v;
    }
    const bool ok = !bad && ((__int128)(long long)H << 40) + (long long)L == exact;
    std::printf("%s slab words\n", ok ? "ok" : "BAD");
    return !ok;
}

int main()
{
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> one(0.5, 1.5), small(0.0, 1.0 / 256.0);
    int bad = words() + slab();
    for (double s : {1.0, -1.0})
    {
        bad += sum("0.003", 300000, [&](long) { return s * 0.003; });
        bad += sum("below 2^-8", 300000, [&](long) { return s * std::nextafter(1.0 / 256.0, 0.0); });
        bad += sum("2^-9", 300000, [&](long) { return s * 0x1p-9; });
        bad += sum("random below 2^-8", 4000000, [&](long) { return s * small(g); });
        bad += sum("random near 1", 1L << 26, [&](long) { return s * one(g); });
    }
    return bad != 0;
}
