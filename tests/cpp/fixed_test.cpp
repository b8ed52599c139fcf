// Host check of fixed64.h and of the tables it reads, against extended precision:
// * the integer split of a double into the accumulators' two words equals the floating form (rint
//   at 2^-20, then at 2^-60) at every exponent it covers, ties included;
// * the inverse normal of every generator's draws;
// * interval, vol and path step on even, uneven and one-knot grids, inside and outside of them.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <random>

#include "fx_tables.h"
#include "host_math.h"

static unsigned long long bits(double v)
{
    unsigned long long b;
    std::memcpy(&b, &v, 8);
    return b;
}

static int split()
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

typedef long double real;  // 64 or more bits on both build hosts

static real bsm(int gen, unsigned up)
{
    const double c = 2.3283064365387E-10;
    const real u = gen == cf::FXG_MRG ? (real)up / 4294967088.0L
                   : gen == cf::FXG_SOBOL_LOWER ? (real)c * up : 1.0L - (real)c * (4294967296.0L - up);
    const double p = gen == cf::FXG_MRG ? up / 4294967088.0 : gen == cf::FXG_SOBOL_LOWER ? c * up : 1.0 - c * (4294967296.0 - up);
    if (std::fabs(p - 0.5) < 0.42)
    {
        const real x = 0.5L - u, r = x * x;
        return x * (((-25.44106049637 * r + 41.39119773534) * r + -18.61500062529) * r + 2.50662823884) /
               ((((3.13082909833 * r + -21.06224101826) * r + 23.08336743743) * r + -8.47351093090) * r + 1.0L);
    }
    const double k[9] = {0.3374754822726147, 0.9761690190917186, 0.1607979714918209, 0.0276438810333863,
                         0.0038405729373609, 0.0003951896511919, 0.0000321767881768, 0.0000002888167364,
                         0.0000003960315187};
    const real r = logl(-logl(u));
    real v = 0.0L;
    for (int i = 8; i >= 0; --i) v = v * r + k[i];
    return v;
}

// Error bound: 2^-55 for the quartic and its roundings, and the reference's own rounding (the
// upper Sobol half subtracts from 1 at 2^-64, a tail's sensitivity is 1 / (u |g|)).
static int gauss(int gen)
{
    std::vector<cf::FxgPiece> t(cf::FXG_PIECES);
    const unsigned brk = cf::inv_normal_table64(gen, t.data());
    const unsigned most = gen == cf::FXG_MRG ? 2147483544u : 1u << 31;
    std::mt19937_64 g(11 + gen);
    long bad = brk == 0, n = 0;
    real sumFx = 0.0L, sumD = 0.0L;
    auto check = [&](unsigned up) {
        if (up < 1 || up > most) return;
        int w;
        const int k = cf::fxg_piece(up, brk, w);
        const real v = ldexpl((real)cf::fxg_value(t[k], w), -cf::FX_G), ref = bsm(gen, up);
        const real own = gen == cf::FXG_SOBOL_UPPER ? ldexpl(1.0L, -63) * 4294967296.0L / up : 0.0L;
        if (k < 0 || k >= cf::FXG_PIECES || !(fabsl(v - ref) <= ldexpl(1.0L, -55) + own)) ++bad;
        const double p = gen == cf::FXG_MRG ? up / 4294967088.0 : gen == cf::FXG_SOBOL_LOWER ? 2.3283064365387E-10 * up
                         : 1.0 - 2.3283064365387E-10 * (4294967296.0 - up);
        if (p < 0.5)
        {
            sumFx += fabsl(v - ref);
            sumD += fabsl(-cf::inv_normal_bsm(p) - ref);
        }
        ++n;
    };
    for (unsigned d = 0; d < 1200; ++d) check(1 + d), check(brk - 600 + d), check(most - d);
    for (int b = 0; b < 32; ++b)
        for (int i = 0; i < 4000; ++i) check((1u << b) + (unsigned)(g() % (1ULL << std::min(b, 30))));
    for (int i = 0; i < 400000; ++i) check(1 + (unsigned)(g() >> 33));
    if (!(sumFx < sumD)) ++bad;  // and on average nearer than the double evaluation
    std::printf("%s inverse normal %d: %ld draws\n", bad ? "BAD" : "ok", gen, n);
    return bad != 0;
}

// Steps of `paths` random paths in fixed point, in doubles as the generic kernel takes them, and in
// extended precision.  The state follows double rounding near log S0, so the fixed-point path may
// be as far from the extended one as a double's: per step one rounding to `grid` (half a unit) and
// the vol's 2^-56, amplified by at most (1 + |g - v| slope) per step.
static int paths(const char* what, double spot, std::vector<double> spots, int steps, double volLevel, int paths, bool fits)
{
    std::mt19937_64 g(5);
    std::normal_distribution<double> gs;
    std::uniform_real_distribution<double> un;
    cf::FxInput in;
    const int nS = int(spots.size());
    in.nSteps = steps;
    in.x0 = std::log(spot);
    std::vector<double> X;
    for (double s : spots) X.push_back(std::log(s)), in.X.push_back(std::log(s) - in.x0);
    const double sq = std::sqrt(3.0 / steps);
    for (int i = 0; i < steps; ++i)
    {
        for (int j = 0; j < nS; ++j) in.Y.push_back(sq * volLevel * (0.8 + 0.4 * un(g)));
        in.sq.push_back(sq);
        in.tw.push_back(un(g));
        in.colA.push_back(0);
        in.colB.push_back(1);
    }
    cf::FxHost h;
    long bad = cf::fx_lower(in, h) != fits, n = 0;
    if (bad || !fits)
    {
        std::printf("%s %s: %s\n", bad ? "BAD" : "ok", what, fits ? "lowered" : "refused");
        return bad != 0;
    }
    const real unitY = ldexpl(1.0L, h.r - cf::FX_Y), unitV = ldexpl(1.0L, h.r - cf::FX_V);
    auto interval = [&](long long y) { return cf::fx_interval(h.bucket.data(), int(h.bucket.size()), h.shift, h.x0h, y); };
    // every knot, its neighbours beyond the packed bits, and random states
    auto where = [&](long long y) {
        const real x = y * unitY;
        int lo = 0;
        while (lo < nS && in.X[lo] <= (double)x) ++lo;
        return lo;
    };
    for (int j = 0; j < nS; ++j)
        for (long long d : {0LL, 5000LL, -9000LL, 1LL << 40, -(1LL << 40)})
        {
            const long long y = llrintl(in.X[j] / unitY) + d;
            if (interval(y) != (d == 0 ? j + 1 : where(y))) ++bad;
        }
    real worst = 0.0L, bound = 0.0L;
    for (int k = 0; k < paths; ++k)
    {
        long long y = 0;
        real x = 0.0L, slack = 0.0L;
        for (int i = 0; i < steps; ++i)
        {
            const long long z = llrint(std::ldexp(std::max(-6.2, std::min(6.2, gs(g))), cf::FX_G));
            const real gz = ldexpl((real)z, -cf::FX_G);
            const int lo = interval(y);
            if (lo < 0 || lo > nS) return std::printf("BAD %s: interval\n", what), 1;
            const cf::FxVol c = h.vol[size_t(i) * (nS + 1) + lo];
            const long long v = cf::fx_vol(c.a, c.bl, c.bh, y, h.center, h.sh);
            // the vol at the fixed-point state, in extended precision
            auto volAt = [&](real s, real& slope) -> real {
                const double* r = &in.Y[size_t(i) * nS];
                slope = 0.0L;
                if (s < in.X[0]) return r[0];
                if (s >= in.X[nS - 1]) return r[nS - 1];
                int q = 1;
                while (in.X[q] <= s) ++q;
                slope = ((real)r[q] - r[q - 1]) / ((real)in.X[q] - in.X[q - 1]);
                return r[q - 1] + slope * (s - in.X[q - 1]);
            };
            real sl, sl2;
            const real ve = volAt(y * unitY, sl);
            if (!(fabsl(v * unitV - ve) <= ldexpl(1.0L, -56) + 4096 * unitY * fabsl(sl) * 2)) ++bad;
            const real vx = volAt(x, sl2);
            x += vx * (gz - 0.5L * vx);
            y = cf::fx_step(y, v, z, h.r, h.grid << 31, h.grid);
            const real amp = 1.0L + fabsl(gz - ve) * std::max(fabsl(sl), fabsl(sl2));
            slack = slack * amp + 0.5L * h.grid * unitY + unitY + ldexpl(1.0L, -56) * (fabsl(gz) + 1.0L) +
                    8192 * unitY * std::max(fabsl(sl), fabsl(sl2)) * (fabsl(gz) + 1.0L) * 0x1p-12L;
            if (!(fabsl(y * unitY - x) <= slack)) ++bad;
            ++n;
        }
        worst = std::max(worst, (real)fabsl(y * unitY - x));
        bound = std::max(bound, slack);
    }
    std::printf("%s %s: %ld steps, r %d, worst %.2Lg of %.2Lg\n", bad ? "BAD" : "ok", what, n, h.r, worst, bound);
    return bad != 0;
}

static int smoothing()
{
    long bad = 0;
    for (int r = 0; r <= 4; ++r)
        for (int k = 0; k <= 1000; ++k)
        {
            const long long w = (long long)(k / 1000.0 * 0.99 * std::ldexp(1.0, cf::FX_Y - r - cf::FX_SMOOTH_BITS));
            const real u = ldexpl((real)w, r - cf::FX_Y), v = ldexpl((real)cf::fx_one_minus_exp8(w, r), -62);
            if (!(fabsl(v + 8.0L * expm1l(-u)) <= ldexpl(1.0L, -59))) ++bad;
        }
    std::printf("%s smoothing factor\n", bad ? "BAD" : "ok");
    return bad != 0;
}

// Relative error: 2^-56 for the sum of the roundings, and the argument's own unit.
static int exponential()
{
    std::vector<long long> t(1 << cf::FX_EXP_BITS);
    cf::exp_table64(t.data());
    std::mt19937_64 g(9);
    long bad = 0;
    auto check = [&](long long a) {
        int n;
        const long long m = cf::fx_exp(t.data(), a, n);
        const real ref = expl(ldexpl((real)a, -cf::FX_A));
        if (m < (1LL << 60) || !(fabsl(ldexpl((real)m, n - 61) / ref - 1.0L) <= ldexpl(1.0L, -56))) ++bad;
    };
    for (int i = 0; i < 300000; ++i) check((long long)(g() >> (1 + g() % 60)) * ((i & 1) ? 1 : -1) % (1LL << 62));
    for (int i = -2000; i <= 2000; ++i)  // around the table's steps
    {
        const long long a = llrintl(ldexpl(i * logl(2.0L) / 256, cf::FX_A));
        check(a), check(a + 1), check(a - 1);
    }
    check(0), check((1LL << 62) - 1), check(-(1LL << 62) + 1);
    std::printf("%s exponential\n", bad ? "BAD" : "ok");
    return bad != 0;
}

int main()
{
    auto even = [](double a, double b, int n) {
        std::vector<double> s;
        for (int i = 0; i < n; ++i) s.push_back(a * std::pow(b / a, n > 1 ? i / double(n - 1) : 0.0));
        return s;
    };
    std::vector<double> uneven;
    for (int i = 0; i < 40; ++i) uneven.push_back(40.0 + 3.0 * i + (i % 7 == 0 ? 0.02 : 1.1));
    int bad = split() + gauss(0) + gauss(1) + gauss(2) + smoothing() + exponential();
    bad += paths("60 knots", 100.0, even(50, 200, 60), 156, 0.2, 300, true);
    bad += paths("120 knots, 520 steps", 100.0, even(50, 200, 120), 520, 0.3, 100, true);
    bad += paths("uneven knots", 100.0, uneven, 36, 0.25, 300, true);
    bad += paths("one knot", 100.0, {80.0}, 12, 0.25, 300, true);
    bad += paths("two knots far apart", 100.0, {1.0, 9000.0}, 12, 0.25, 300, true);
    bad += paths("spot 1.1", 1.1, even(0.5, 2.0, 60), 52, 0.2, 300, true);
    bad += paths("spot below the grid", 20.0, even(50, 200, 60), 52, 0.2, 300, true);
    bad += paths("spot 1e5 above the grid", 1e5, even(50, 200, 60), 52, 0.2, 300, true);
    bad += paths("large vols", 100.0, even(50, 200, 20), 12, 1.5, 300, true);
    bad += paths("vols beyond the range", 100.0, even(50, 200, 20), 12, 40.0, 1, false);
    bad += paths("knots too close", 100.0, {99.0, 100.0, 100.0 + 1e-9}, 12, 0.2, 1, false);
    bad += paths("knots out of order", 100.0, {100.0, 90.0}, 12, 0.2, 1, false);
    return bad != 0;
}
