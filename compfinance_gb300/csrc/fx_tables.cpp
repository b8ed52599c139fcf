// Lowering of a Dupire plan to fixed point (fx_tables.h).
#include "fx_tables.h"

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "host_math.h"

namespace cf {

namespace {

// Largest Gaussian of the generators' draws (the smallest uniform, 2.3e-10, gives 6.24).
constexpr double kMaxGauss = 6.3;

// d 2^k / w to the nearest, halves away from zero, for one w and many d.  A 128-bit division for each took most
// of a model's lowering (60x30 grid, 156 steps: 0.35 -> 0.13 ms; 120x60, 520 steps: 2.4 -> 0.9 ms); two
// steps by the rounded reciprocal leave a remainder that at most one correction brings into [0, w).
struct Quotient
{
    long long w = 1;
    int k = 0;
    double inv = 1.0, invK = 1.0;  // 1 / w, 2^k / w
    void set(long long width, int bits)
    {
        w = width;
        k = bits;
        inv = 1.0 / double(w);
        invK = std::ldexp(inv, k);
    }
    // false when the quotient is not below limit (at most 2^63) in magnitude
    bool divide(long long d, double limit, long long& q) const
    {
        const double e = std::fabs(double(d)) * invK;
        if (!(e < limit)) return false;
        const unsigned long long m = d < 0 ? 0ULL - (unsigned long long)d : (unsigned long long)d;
        long long b = (long long)e - 4096;  // below the quotient: e is within 2^-51 of it, 2^12 at most
        __int128 r = (__int128)(((unsigned __int128)m << k) + (unsigned long long)(w / 2)) - (__int128)b * w;
        const double rd = double((long long)(r >> 64)) * 0x1p64 + double((unsigned long long)r);
        const long long c = (long long)(rd * inv);
        r -= (__int128)c * w;
        b += c;
        for (; r < 0; r += w) --b;
        for (; r >= w; r -= w) ++b;
        q = d < 0 ? -b : b;
        return true;
    }
};

// The tables with r bits of range: 1 done, 0 a magnitude needs more bits, -1 none would do.
int lower_with(const FxInput& in, double reach, int r, FxHost& h)
{
    const int nS = int(in.X.size()), n = in.nSteps, sy = FX_Y - r, sv = FX_V - r;
    const std::vector<double>&X = in.X, &Y = in.Y;
    if (std::ldexp(1.0, 4 + r) < reach) return 0;
    h = FxHost();
    h.r = r;
    h.nSteps = n;
    h.nS = nS;
    const int ulp = in.x0 != 0.0 ? std::ilogb(in.x0) - 52 + sy : 0;  // a double's unit near log S0
    h.grid = 1LL << std::max(0, std::min(ulp, 30));
    std::vector<long long> K(nS);
    for (int j = 0; j < nS; ++j) K[j] = std::llrint(std::ldexp(X[j], sy));
    // buckets: the widest power of two not above the smallest gap, the first edge below the first knot
    long long gap = 1LL << sy;
    for (int j = 0; j + 1 < nS; ++j) gap = std::min(gap, K[j + 1] - K[j]);
    int wb = 62;
    while (wb >= 33 && (1LL << wb) > gap) --wb;
    if (gap <= 0 || wb < 33 || nS >= (1 << FX_LO_BITS)) return -1;
    h.shift = wb - 32;
    h.x0h = int((K[0] - (1LL << (wb - 1))) >> 32);
    const long long x0 = (long long)h.x0h * (1LL << 32), nB = ((K[nS - 1] - x0) >> wb) + 2;
    if (nB > 4096) return -1;
    constexpr long long loMask = (1LL << FX_LO_BITS) - 1;
    for (long long b = 0; b < nB; ++b)
    {
        const int lo = int(std::upper_bound(K.begin(), K.end(), x0 + (b << wb)) - K.begin());
        // at most the knot: a state on it (today's spot, often) belongs to the interval above
        h.bucket.push_back((((lo < nS ? K[lo] : INT64_MAX) - loMask) & ~loMask) | lo);
    }
    const double most = std::ldexp(0.999, 62);  // of a vol; slopes and D may use another bit
    h.center = (K[0] + K[nS - 1]) / 2;
    if (nS > 1)
        while (h.sh < 40 && std::ldexp(double((K[nS - 1] - K[0]) / 2 + 1), h.sh + 1) < 2 * most) ++h.sh;
    h.interval.assign(size_t(nS) + 1, FxInterval{0, 0, 0});
    h.inv.assign(size_t(nS) + 1, 0);
    for (int lo = 1; lo < nS; ++lo)
    {
        const long long d = K[lo] - K[lo - 1];
        int sh = 0;
        while (d < (1LL << (61 - sh))) ++sh;  // d 2^sh in [2^61, 2^62)
        h.interval[lo] = FxInterval{K[lo - 1], sh, 0};
        h.inv[lo] = (long long)(((unsigned __int128)1 << 123) / (unsigned long long)(d << sh));
    }
    h.vol.resize(size_t(n) * (nS + 1));
    h.slope.assign(size_t(n) * (nS + 1), 0.0);
    h.step.reserve(n);
    const __int128 mostI = (long long)most;
    const double scale = std::ldexp(1.0, sv), unit = std::ldexp(1.0, -FX_G);
    std::vector<Quotient> width(nS);  // by the interval's width, for slopes in units 2^64 / 2^sh per state unit
    for (int lo = 1; lo < nS; ++lo) width[lo].set(K[lo] - K[lo - 1], 64 - h.sh);
    for (int i = 0; i < n; ++i)
    {
        FxVol* o = &h.vol[size_t(i) * (nS + 1)];
        double* slope = &h.slope[size_t(i) * (nS + 1)];
        const double* y = &Y[size_t(i) * nS];
        for (int j = 0; j < nS; ++j)
            if (!(std::fabs(y[j] * scale) < most)) return 0;
        long long a = std::llrint(y[0] * scale);
        o[0] = FxVol{a, 0, 0};
        for (int lo = 1; lo < nS; ++lo)
        {
            // slope b to the nearest; value at the center
            const long long next = std::llrint(y[lo] * scale), d = next - a;
            long long b;
            if (!width[lo].divide(d, 2 * most, b)) return 0;
            const __int128 off = (__int128)b * ((h.center - K[lo - 1]) * (1LL << h.sh));
            const __int128 at = (__int128)a + ((off + ((__int128)1 << 63)) >> 64);
            if (at >= mostI || at <= -mostI) return 0;
            const int bl = int(unsigned((unsigned long long)b));
            o[lo] = FxVol{(long long)at, bl, int((b - bl) >> 32)};
            slope[lo] = (y[lo] - y[lo - 1]) / (X[lo] - X[lo - 1]) * unit;
            a = next;
        }
        o[nS] = FxVol{a, 0, 0};
        h.step.push_back(FxStep{std::llrint(std::ldexp(in.tw[i], 62)), in.sq[i], in.colA[i] * in.node.c,
                                in.colB[i] * in.node.c, in.colA[i], in.colB[i]});
    }
    return 1;
}

}  // namespace

bool fx_lower(const FxInput& in, FxHost& h)
{
    const int nS = int(in.X.size()), n = in.nSteps;
    double reach = 1.0;  // bound of |log S - log S0| and of the knots
    for (int i = 0; i < n; ++i)
    {
        double vMax = 0.0;
        for (int j = 0; j < nS; ++j)
        {
            const double v = std::fabs(in.Y[size_t(i) * nS + j]);
            if (!(v < 16.0)) return false;
            vMax = std::max(vMax, v);
        }
        reach += vMax * (kMaxGauss + 0.5 * vMax);
    }
    for (double x : in.X)
    {
        if (!(std::fabs(x) < 200.0)) return false;
        reach = std::max(reach, 1.0 + std::fabs(x));
    }
    for (int r = 0, got = 0; r <= 4; ++r)
        if ((got = lower_with(in, reach, r, h)) != 0) return got > 0;
    return false;
}

long long fx_state(double level, double logSpot, int r)
{
    if (!(level > 0.0)) return INT64_MIN;
    if (std::isinf(level)) return INT64_MAX;
    double hi, lo;
    log_dd(level, hi, lo);
    // hi - logSpot as the rounded difference d and its error (Knuth's two-sum)
    const double d = hi - logSpot, t = d - hi;
    lo += (hi - (d - t)) - (logSpot + t);
    const double v = std::ldexp(d, FX_Y - r), w = std::ldexp(lo, FX_Y - r);
    if (!(v > -9.2e18)) return INT64_MIN;
    if (!(v < 9.2e18)) return INT64_MAX;
    const double f = std::floor(v);
    return (long long)f + (long long)std::floor((v - f) + w);
}

}  // namespace cf
