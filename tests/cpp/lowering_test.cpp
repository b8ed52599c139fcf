// Host check of fx_lower's vols and slopes (fx_tables.h): every table entry against whole-number division of
// 128 bits, over grids and vols of every range; and its time against those divisions alone.
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

#include "fx_tables.h"

static cf::FxInput model(int nS, int n, double lo, double hi, double vol, bool even, unsigned seed)
{
    std::mt19937_64 g(seed);
    std::uniform_real_distribution<double> un(0.0, 1.0);
    cf::FxInput in;
    in.nSteps = n;
    in.x0 = std::log(100.0);
    for (int j = 0; j < nS; ++j)
        in.X.push_back(std::log(lo * std::pow(hi / lo, nS > 1 ? (j + (even ? 0.0 : 0.8 * un(g))) / nS : 0.0)) - in.x0);
    for (int i = 0; i < n; ++i)
    {
        for (int j = 0; j < nS; ++j) in.Y.push_back(vol * (j % 7 == 3 ? 0.0 : j % 5 == 1 ? -un(g) : un(g)));
        in.sq.push_back(0.1);
        in.tw.push_back(un(g));
        in.colA.push_back(0);
        in.colB.push_back(1);
    }
    return in;
}

// The slope of interval lo in step i, to the nearest, halves away from zero.
static long long slope(const cf::FxInput& in, const cf::FxHost& h, int i, int lo)
{
    const int nS = h.nS, sv = cf::FX_V - h.r, sy = cf::FX_Y - h.r;
    const double* y = &in.Y[size_t(i) * nS];
    const long long a = std::llrint(std::ldexp(y[lo - 1], sv)), d = std::llrint(std::ldexp(y[lo], sv)) - a;
    const long long w = std::llrint(std::ldexp(in.X[lo], sy)) - std::llrint(std::ldexp(in.X[lo - 1], sy));
    const __int128 num = (__int128)d * ((__int128)1 << (64 - h.sh));
    return (long long)((num + (num < 0 ? -w : w) / 2) / w);
}

static int tables(const char* what, const cf::FxInput& in, int range)
{
    cf::FxHost h;
    if (!cf::fx_lower(in, h)) return std::printf("BAD %s: refused\n", what), 1;
    long bad = h.r != range;
    const int nS = h.nS;
    for (int i = 0; !bad && i < h.nSteps; ++i)
    {
        const double* y = &in.Y[size_t(i) * nS];
        const cf::FxVol* o = &h.vol[size_t(i) * (nS + 1)];
        const double* s = &h.slope[size_t(i) * (nS + 1)];
        auto fx = [&](int j) { return std::llrint(std::ldexp(y[j], cf::FX_V - h.r)); };
        if (o[0].a != fx(0) || o[0].bl || o[0].bh || o[nS].a != fx(nS - 1) || o[nS].bl || o[nS].bh || s[0] || s[nS]) ++bad;
        for (int lo = 1; lo < nS; ++lo)
        {
            const long long b = slope(in, h, i, lo), k = std::llrint(std::ldexp(in.X[lo - 1], cf::FX_Y - h.r));
            const __int128 off = (__int128)b * ((h.center - k) * (1LL << h.sh));
            const long long a = (long long)((__int128)fx(lo - 1) + ((off + ((__int128)1 << 63)) >> 64));
            if (((long long)o[lo].bh * (1LL << 32)) + o[lo].bl != b || o[lo].a != a) ++bad;
            if (s[lo] != (y[lo] - y[lo - 1]) / (in.X[lo] - in.X[lo - 1]) * std::ldexp(1.0, -cf::FX_G)) ++bad;
        }
    }
    std::printf("%s %s: r %d\n", bad ? "BAD" : "ok", what, h.r);
    return bad != 0;
}

template <class F>
static double best(F&& f)
{
    double t = 1e9;
    for (int k = 0; k < 40; ++k)
    {
        const auto t0 = std::chrono::steady_clock::now();
        f();
        t = std::min(t, std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count());
    }
    return t;
}

int main(int argc, char**)
{
    int bad = 0;
    bad += tables("60 knots", model(60, 156, 50, 200, 0.02, true, 1), 1);
    bad += tables("20 knots", model(20, 12, 50, 200, 0.1, true, 1), 2);
    bad += tables("120 uneven knots", model(120, 260, 30, 300, 0.002, false, 2), 0);
    bad += tables("two knots", model(2, 12, 50, 200, 0.3, true, 3), 0);
    bad += tables("one knot", model(1, 3, 50, 200, 0.3, true, 4), 0);
    bad += tables("steep", model(300, 12, 50, 200, 0.003, true, 5), 1);
    bad += tables("wide range", model(40, 520, 1, 9000, 0.03, false, 6), 3);
    bad += tables("wide and steep", model(100, 520, 1, 9000, 0.05, true, 6), 4);
    if (argc > 1)
    {
        const cf::FxInput in = model(120, 520, 50, 200, 0.02, true, 7);
        cf::FxHost h;
        cf::fx_lower(in, h);
        volatile long long sink = 0;
        const double div = best([&] {
            for (int i = 0; i < 520; ++i)
                for (int lo = 1; lo < 120; ++lo) sink = sink + slope(in, h, i, lo);
        });
        const double low = best([&] {
            cf::FxHost g;
            cf::fx_lower(in, g);
        });
        std::printf("%s lowering %.2f ms, its divisions alone %.2f ms\n", low < 0.65 * div ? "ok" : "BAD", low * 1e3, div * 1e3);
        bad += !(low < 0.65 * div);
    }
    return bad != 0;
}
