// Host check of one fixed-point path step at a time (fixed64.h, fx_tables.h): from the same state, vol and next
// state against extended precision, with a bound that does not grow along the path.  Smooth and rough
// vols, states inside and outside of the grid, on knots and next to them.
#include <cmath>
#include <cstdio>
#include <random>

#include "fx_tables.h"

typedef long double real;  // 64 or more bits on both build hosts

static int steps(const char* what, double spot, int nS, double lo, double hi, double level, bool rough, int n)
{
    std::mt19937_64 g(6);
    std::uniform_real_distribution<double> un(0.0, 1.0);
    std::normal_distribution<double> gs;
    cf::FxInput in;
    in.nSteps = n;
    in.x0 = std::log(spot);
    for (int j = 0; j < nS; ++j) in.X.push_back(std::log(lo * std::pow(hi / lo, nS > 1 ? j / double(nS - 1) : 0.0)) - in.x0);
    for (int i = 0; i < n; ++i)
    {
        for (int j = 0; j < nS; ++j)
            in.Y.push_back(level * (rough ? 0.8 + 0.4 * un(g) : 1.0 + 0.5 * in.X[j] * in.X[j] / (1.0 + in.X[j] * in.X[j])));
        in.sq.push_back(0.1);
        in.tw.push_back(0.5);
        in.colA.push_back(0);
        in.colB.push_back(0);
    }
    cf::FxHost h;
    if (!cf::fx_lower(in, h)) return std::printf("BAD %s: refused\n", what), 1;
    const real unitY = ldexpl(1.0L, h.r - cf::FX_Y), unitV = ldexpl(1.0L, h.r - cf::FX_V), unitG = ldexpl(1.0L, -cf::FX_G);
    long bad = 0, count = 0;
    real worst = 0.0L;
    auto check = [&](int i, long long y) -> long long {
        const int k = cf::fx_interval(h.bucket.data(), int(h.bucket.size()), h.shift, h.x0h, y);
        const cf::FxVol c = h.vol[size_t(i) * (nS + 1) + k];
        const long long z = llrint(std::ldexp(std::max(-6.2, std::min(6.2, gs(g))), cf::FX_G));
        const long long v = cf::fx_vol(c.a, c.bl, c.bh, y, h.center, h.sh);
        // the vol between the knots around the state: interval q has knots q - 1 and q, the flat ends one
        const real x = y * unitY;
        const double* r = &in.Y[size_t(i) * nS];
        auto slope = [&](int q) -> real {
            return q > 0 && q < nS ? ((real)r[q] - r[q - 1]) / ((real)in.X[q] - in.X[q - 1]) : 0.0L;
        };
        int q = 0;
        while (q < nS && in.X[q] <= x) ++q;
        const int knot = q > 0 ? q - 1 : 0;
        const real ve = r[knot] + slope(q) * (x - in.X[knot]);
        // knots are rounded to the state's unit; the line's value, its slope and their product to a unit of the
        // vol's each; an interval may begin 2^13 units early, where the vol is the next one's line
        real tolV = 4.0L * unitV + fabsl(slope(q)) * unitY;
        for (int j = 0; j < nS; ++j)
            if (fabsl(in.X[j] - x) <= 16384 * unitY) tolV += (fabsl(slope(j)) + fabsl(slope(j + 1))) * 8192 * unitY;
        if (!(fabsl(v * unitV - ve) <= tolV)) ++bad;
        const real vf = v * unitV, gz = z * unitG;
        const long long next = cf::fx_step(y, v, z, h.r, h.grid << 31, h.grid);
        // half a unit of the grid, one of the state for the product, and half a unit of the Gaussian for v / 2
        const real exact = x + vf * (gz - 0.5L * vf), err = fabsl(next * unitY - exact);
        if (!(err <= 0.5L * h.grid * unitY + unitY + fabsl(vf) * unitG) || next % h.grid) ++bad;
        worst = std::max(worst, err / (h.grid * unitY));
        ++count;
        return next;
    };
    for (int p = 0; p < 300; ++p)
    {
        long long y = 0;
        for (int i = 0; i < n; ++i) y = check(i, y);
    }
    for (int j = 0; j < nS; ++j)
        for (long long d : {0LL, 1LL << 13, -(1LL << 13), 1LL << 40, -(1LL << 40)})
            check(j % n, (llrintl(in.X[j] / unitY) + d) & -h.grid);
    std::printf("%s %s: %ld steps, r %d, worst %.3Lf grid units\n", bad ? "BAD" : "ok", what, count, h.r, worst);
    return bad != 0;
}

int main()
{
    int bad = 0;
    bad += steps("60 knots", 100.0, 60, 50, 200, 0.015, false, 156);
    bad += steps("60 rough knots", 100.0, 60, 50, 200, 0.015, true, 156);
    bad += steps("120 knots, 520 steps", 100.0, 120, 50, 200, 0.015, false, 520);
    bad += steps("120 rough knots, 520 steps", 100.0, 120, 50, 200, 0.015, true, 520);
    bad += steps("one knot", 100.0, 1, 80, 80, 0.1, false, 12);
    bad += steps("large vols", 100.0, 20, 50, 200, 0.7, false, 12);
    bad += steps("spot 1.1", 1.1, 60, 0.5, 2.0, 0.03, false, 52);
    bad += steps("far above the grid", 1e5, 60, 50, 200, 0.03, true, 52);
    bad += steps("far below the grid", 0.01, 60, 50, 200, 0.03, false, 52);
    return bad != 0;
}
