// Tables of the fixed-point exponential and inverse normal (fixed64.h), the latter Beasley-Springer-Moro (gaussians.h:47-87)
// evaluated in double-double arithmetic at five Chebyshev nodes of every piece.  The tables are
// built once per context.  Compiled with -ffp-contract=off.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <future>

#include "host_math.h"

namespace cf {

namespace {

struct DD  // hi + lo, |lo| <= ulp(hi) / 2
{
    double hi, lo;
    DD(double h = 0.0, double l = 0.0) : hi(h), lo(l) {}
};
inline DD fast_two(double a, double b)
{
    const double s = a + b;
    return DD(s, b - (s - a));
}
inline DD operator+(const DD& a, const DD& b)
{
    const double s = a.hi + b.hi, t = s - a.hi;
    const double e = (a.hi - (s - t)) + (b.hi - t);
    return fast_two(s, e + a.lo + b.lo);
}
inline DD operator-(const DD& a) { return DD(-a.hi, -a.lo); }
inline DD operator-(const DD& a, const DD& b) { return a + (-b); }
inline DD operator*(const DD& a, const DD& b)
{
    const double p = a.hi * b.hi, e = std::fma(a.hi, b.hi, -p);
    return fast_two(p, e + (a.hi * b.lo + a.lo * b.hi));
}
inline DD operator/(const DD& a, const DD& b)
{
    const double q1 = a.hi / b.hi;
    const DD r = a - b * DD(q1);
    const double q2 = r.hi / b.hi;
    const DD r2 = r - b * DD(q2);
    return fast_two(q1, q2) + DD(r2.hi / b.hi);
}

// log x: the double logarithm y0, corrected by the series of log(1 + d) at d = x exp(-y0) - 1.
// exp(-y0) = 2^k E(r / 64)^64 with the Taylor series of E.
DD dd_log(const DD& x)
{
    static const DD ln2(6.931471805599452862e-01, 2.319046813846299558e-17);
    const double y0 = std::log(x.hi);
    const double k = std::nearbyint(-y0 / ln2.hi);
    const DD r = DD(-y0) - DD(k) * ln2;
    const DD s(r.hi / 64.0, r.lo / 64.0);  // |s| < 0.0055
    // E - 1 = s + s^2/2 + ...; terms from the fourth on are below 2^-32 of the first: doubles do
    DD sum = s;
    DD t = s * s;
    sum = sum + DD(0.5 * t.hi, 0.5 * t.lo);
    t = t * s / DD(6.0);
    sum = sum + t;
    t = t * s * DD(0.25);
    sum = sum + t;
    double u = t.hi * s.hi / 5.0;
    double rest = u;
    for (int i = 6; i < 12; ++i) rest += (u *= s.hi / i);
    sum = sum + DD(rest);
    for (int i = 0; i < 6; ++i) sum = sum * DD(2.0) + sum * sum;  // (1 + q)^2 - 1
    const DD e = sum + DD(1.0);
    const DD z = x * DD(std::ldexp(e.hi, int(k)), std::ldexp(e.lo, int(k)));
    const DD d = z - DD(1.0);  // of the order of a double's rounding
    return DD(y0) + d - DD(0.5 * d.hi * d.hi);
}

const double kA[4] = {2.50662823884, -18.61500062529, 41.39119773534, -25.44106049637};
const double kB[4] = {-8.47351093090, 23.08336743743, -21.06224101826, 3.13082909833};
const double kC[9] = {0.3374754822726147, 0.9761690190917186, 0.1607979714918209, 0.0276438810333863,
                      0.0038405729373609, 0.0003951896511919, 0.0000321767881768, 0.0000002888167364,
                      0.0000003960315187};

DD central(const DD& u)  // |u - 0.5| < 0.42: the distance of the value from zero (u below 1/2)
{
    const DD x = DD(0.5) - u, r = x * x;
    DD n(kA[3]), d(kB[3]);
    for (int i = 2; i >= 0; --i)
    {
        n = n * r + DD(kA[i]);
        d = d * r + DD(kB[i]);
    }
    return x * n / (d * r + DD(1.0));
}

DD tail(const DD& logu)
{
    const DD r = dd_log(-logu);
    DD s(kC[8]);
    for (int i = 7; i >= 0; --i) s = s * r + DD(kC[i]);
    return s;
}

long long to_fixed(const DD& v, int shift)
{
    return llrint(std::ldexp(v.hi, shift)) + llrint(std::ldexp(v.lo, shift));
}

}  // namespace

void log_dd(double x, double& hi, double& lo)
{
    const DD l = dd_log(DD(x));
    hi = l.hi;
    lo = l.lo;
}

void exp_table64(long long* out)
{
    // 2^(1/128) by seven square roots of 2 (Newton steps of r - (r^2 - a) / (2 r)), then its powers
    DD root(2.0);
    for (int k = 0; k < FX_EXP_BITS; ++k)
    {
        DD r(std::sqrt(root.hi));
        for (int i = 0; i < 2; ++i) r = r - (r * r - root) / (r + r);
        root = r;
    }
    DD p(1.0);
    for (int i = 0; i < (1 << FX_EXP_BITS); ++i, p = p * root) out[i] = to_fixed(p, 61);
}

unsigned inv_normal_table64(int gen, FxgPiece* out)
{
    // u as a function of the draw's distance up from the end of the range
    const DD inv = DD(1.0) / DD(4294967088.0);
    const double c = 2.3283064365387E-10;  // sobol.h:26, truncated 2^-32
    const DD delta = DD(4294967296.0 * c) - DD(1.0);
    auto uOf = [&](const DD& up) {
        if (gen == FXG_MRG) return up * inv;
        return gen == FXG_SOBOL_LOWER ? up * DD(c) : up * DD(c) - delta;
    };
    const DD logScale = gen == FXG_MRG ? -dd_log(DD(4294967088.0)) : dd_log(DD(c));
    static const DD ln2(6.931471805599452862e-01, 2.319046813846299558e-17);
    // the first draw of the central formula: |u - 0.5| < 0.42 in the reference's double arithmetic
    auto isCentral = [&](double up) {
        const double p = gen == FXG_MRG ? up / 4294967088.0 : gen == FXG_SOBOL_LOWER ? c * up : 1.0 - c * (4294967296.0 - up);
        return std::fabs(p - 0.5) < 0.42;
    };
    unsigned brk = 0;
    for (unsigned step = 1u << 30; step; step >>= 1)
        if (!isCentral(double(brk + step))) brk += step;
    ++brk;
    // five Chebyshev nodes of [0, 1): coefficients up to order 4 from the values by the inverse Vandermonde
    // matrix (rows by Lagrange polynomials)
    constexpr int N = 5;
    double z[N];
    DD M[N][N];  // M[k][j]: coefficient k of the Lagrange polynomial of node j
    for (int j = 0; j < N; ++j)
        z[j] = 0.5 - 0.5 * std::cos((2 * j + 1) * 3.14159265358979323846 / (2 * N));
    for (int j = 0; j < N; ++j)
    {
        DD p[N] = {DD(1.0)};
        int deg = 0;
        for (int i = 0; i < N; ++i)
        {
            if (i == j) continue;
            const DD s = DD(1.0) / (DD(z[j]) - DD(z[i]));
            for (int k = ++deg; k >= 0; --k) p[k] = ((k ? p[k - 1] : DD()) - DD(z[i]) * (k < deg ? p[k] : DD())) * s;
        }
        for (int k = 0; k < N; ++k) M[k][j] = p[k];
    }
    constexpr int nSub = 1 << FXG_SUB_BITS;
    std::vector<DD> logMant(size_t(nSub) * N);  // log of 1 + (sub + z) / nSub, the same in every binade
    for (int sub = 0; sub < nSub; ++sub)
        for (int j = 0; j < N; ++j) logMant[size_t(sub) * N + j] = dd_log(DD(1.0) + (DD(sub) + DD(z[j])) * DD(1.0 / nSub));
    auto value = [&](int b, int sub, int j, bool mid) {  // at node j of the piece; j < 0: at its start
        DD up = DD(1.0) + (DD(sub) + DD(j < 0 ? 0.0 : z[j])) * DD(1.0 / nSub);
        up = DD(std::ldexp(up.hi, b), std::ldexp(up.lo, b));
        if (mid) return central(uOf(up));
        DD lg = (j < 0 ? dd_log(DD(1.0) + DD(sub) * DD(1.0 / nSub)) : logMant[size_t(sub) * N + j]) + DD(b) * ln2 + logScale;
        if (gen == FXG_SOBOL_UPPER)
        {
            const DD e = -(delta / (up * DD(c)));  // log(1 + e), |e| < 8e-6
            lg = lg + e - e * e * DD(0.5) + e * e * e * (DD(1.0) / DD(3.0));
        }
        return tail(lg);
    };
    auto fit = [&](int b, int sub, bool mid, bool& ok) {
        FxgPiece r{0, 0, 0, 0, 0};
        if (b <= FXG_SUB_BITS || b == 31)  // one draw at the piece's start, or none
        {
            if ((sub & ((nSub >> std::min(b, FXG_SUB_BITS)) - 1)) == 0 && (b < 31 || sub == 0))
                r.c0 = to_fixed(value(b, sub, -1, mid), FX_G);
            return r;
        }
        DD y[N];
        for (int j = 0; j < N; ++j) y[j] = value(b, sub, j, mid);
        // the entries of M reach 10^3: the sums cancel, so they are taken in double-double
        double k[N];
        for (int q = 0; q < N; ++q)
        {
            DD t;
            for (int j = 1; j < N; ++j) t = t + M[q][j] * (y[j] - y[0]);
            k[q] = t.hi;
        }
        // variable w / 2^32 = z / 2: coefficient q times 2^q
        r.c0 = to_fixed(y[0] + DD(k[0]), FX_G);
        r.c1 = llrint(std::ldexp(k[1], FX_G + 1));
        r.c2 = llrint(std::ldexp(k[2], FX_G + 2));
        const long long c3 = llrint(std::ldexp(k[3], 55 + 3)), c4 = llrint(std::ldexp(k[4], 55 + 4));
        ok = ok && std::llabs(c3) < (1LL << 30) && std::llabs(c4) < (1LL << 30);
        r.c3 = int(c3);
        r.c4 = int(c4);
        return r;
    };
    const int bBrk = 31 - __builtin_clz(brk);
    const int pBrk = (bBrk << FXG_SUB_BITS) + int(((brk << (31 - bBrk)) >> (31 - FXG_SUB_BITS)) & unsigned(nSub - 1));
    // every piece is on its own: four threads, or this one where no other can be had
    constexpr int PARTS = 4;
    auto part = [&](int first) {
        bool ok = true;
        for (int p = first; p < FXG_PIECES - 1; p += PARTS)
        {
            const int b = p >> FXG_SUB_BITS, sub = p & (nSub - 1);
            if (p <= pBrk) out[p] = fit(b, sub, false, ok);
            if (p >= pBrk) out[p + 1] = fit(b, sub, true, ok);
        }
        return ok;
    };
    std::future<bool> others[PARTS - 1];
    for (int k = 1; k < PARTS; ++k) others[k - 1] = std::async(part, k);
    bool ok = part(0);
    for (std::future<bool>& f : others) ok = f.get() && ok;
    return ok ? brk : 0;
}

}  // namespace cf
