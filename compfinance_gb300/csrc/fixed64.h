// 64-bit integer arithmetic of the fixed-point sums and of the FP64 path kernels' fixed-point form,
// for device code and its host tests.
//
// GB300 executes an FP64 operation at 1/64 of its FP32 rate: a warp's double multiply-add holds its
// SM's FP64 pipe for 16 cycles.  A rounded 64 x 64-bit product by 32-bit multiply-adds takes 6,
// an addition, comparison or table index below 1.  So a path step in 64-bit fixed point, with as
// many fraction bits as a double has at its magnitude or more, costs a fraction of one in doubles.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CF_HD __host__ __device__ __forceinline__
#else
#define CF_HD inline
#endif

namespace cf {

// Upper word of the double word (hi, lo) shifted left, lower word of it shifted right, by 0 <= s < 32.
CF_HD unsigned funnel_left(unsigned lo, unsigned hi, int s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(lo, hi, s);
#else
    return (unsigned)(((((unsigned long long)hi << 32) | lo) << s) >> 32);
#endif
}
CF_HD unsigned funnel_right(unsigned lo, unsigned hi, int s)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_r(lo, hi, s);
#else
    return (unsigned)((((unsigned long long)hi << 32) | lo) >> s);
#endif
}

// A 96-bit word n2 2^64 + n1 2^32 + n0 of units of 2^-60 as hi 2^-20 + lo 2^-60, -2^39 <= lo < 2^39: of either
// sign, so that a sum of low words grows with the root of the number of terms (or, for equal terms, to
// 2^62 in 2^23 of them), not by 2^39 with each.  The value's own low 40 bits have its sign: in one pair
// of words 2^24 terms of one sign, or flushes of a node slab, added up to 2^63.
CF_HD void fix_split_slab(unsigned n0, unsigned n1, unsigned n2, long long& hi, long long& lo)
{
    const int top = (int)(n1 << 24) >> 24;  // bits 32 to 39, signed
    lo = (long long)(((unsigned long long)(unsigned)top << 32) | n0);
    hi = ((long long)(((unsigned long long)n2 << 32) | n1) >> 8) + (top < 0 ? 1 : 0);
}

// The double with bits b as hi 2^-20 + lo 2^-60, rounded to units of 2^-60 (ties to even), |lo| <= 2^39 as
// above; false when |v| >= 2^42 (infinities and NaN included), which the caller converts in floating
// point.  The mantissa is shifted in 32-bit words, as 64-bit shifts by a variable are several instructions each:
// the 60x30 barrier's FP64 risk of 2^18 paths takes 590 us and the four-asset basket's 155, with them 596 and 162.
CF_HD bool fix_split_bits(unsigned long long b, long long& hi, long long& lo)
{
    const unsigned bh = (unsigned)(b >> 32);
    const int E = (int)(bh >> 20) & 0x7ff;
    if (E >= 1023 + 42) return false;
    unsigned m0 = (unsigned)b, m1 = (bh & 0xfffffu) | 0x100000u;
    int sh = E - 1015;  // |v| 2^60 = (m1 2^32 + m0) 2^sh
    if (sh < 0)
    {
        // below 2^-8: shifted right and rounded (zero and subnormals to zero)
        unsigned long long l = 0;
        if (sh >= -54)
        {
            const unsigned long long m = ((unsigned long long)m1 << 32) | m0, half = 1ULL << (-sh - 1), rem = m & (2 * half - 1);
            l = m >> -sh;
            l += (rem > half || (rem == half && (l & 1))) ? 1 : 0;
        }
        m0 = (unsigned)l;
        m1 = (unsigned)(l >> 32);
        sh = 0;
    }
    const int s = sh & 31;  // sh is below 50
    unsigned n0 = m0 << s, n1 = funnel_left(m0, m1, s), n2 = funnel_left(m1, 0, s), n3 = 0;
    if (sh >= 32)
    {
        n3 = n2;
        n2 = n1;
        n1 = n0;
        n0 = 0;
    }
    const int top = (int)(n1 << 24) >> 24;
    lo = (long long)(((unsigned long long)(unsigned)top << 32) | n0);
    hi = (long long)(((unsigned long long)funnel_right(n2, n3, 8) << 32) | funnel_right(n1, n2, 8)) + (top < 0 ? 1 : 0);
    if ((int)bh < 0)
    {
        hi = -hi;
        lo = -lo;
    }
    return true;
}

// c + a b / 2^64, rounded.  The low words enter as signed halves, so their product, at most a
// quarter of the unit, is left out without a bias (error below 0.76 units).  |a|, |b| < 2^62.99.
// half: the rounding constant, 1/2 in units of 2^-32 of the result's unit.
CF_HD long long fx_mul_add(long long a, long long b, long long c, long long half = 0x80000000LL)
{
    const int al = (int)(unsigned)a, bl = (int)(unsigned)b;
    const int ah = (int)((a - al) >> 32), bh = (int)((b - bl) >> 32);
    const long long mid = (long long)ah * bl + (long long)al * bh + half;
    return c + (long long)ah * bh + (mid >> 32);
}

// (s w) / 2^32 for 0 <= w < 2^31, rounded down.
CF_HD long long fx_mul32(long long s, int w)
{
    return (s >> 32) * w + (long long)(((unsigned long long)(unsigned)s * (unsigned)w) >> 32);
}

// ---------------------------------------------------------------------------------------
// Dupire path in fixed point.  The state is y = log S - log S0 in units of 2^-(57 - r), the vols
// sqrt(dt) sigma in 2^-(62 - r), Gaussians in 2^-59; r (0 to 4) is the smallest that holds the bound
// of |y| over all paths, the vols and their slopes.  Between knots a vol is a + b D, with
// D = (y - center) 2^sh scaled so that the grid's half span fills 63 bits; at the flat ends b = 0.
// ---------------------------------------------------------------------------------------
constexpr int FX_Y = 57, FX_V = 62, FX_G = 59;
// A bucket is no wider than the smallest gap between knots, so it holds at most one.  Its entry is
// the first knot above its left edge with the number of knots up to the edge in the low bits (for
// that it moves down by less than 2^13 units; the vol is continuous there).
constexpr int FX_LO_BITS = 12;
struct alignas(16) FxInterval  // between knots lo - 1 and lo; the flat ends have all zero
{
    long long x;
    int sh;
    int unused;
};
// A reverse sweep's node slab in shared memory: node (l, c) of spot l and time column c is at
// l strideL + c strideC.  The lanes of a warp add at one step, so to one column, at intervals l next to
// each other: by spot row (nT, 1) they meet in 32 / gcd(nT, 32) banks, by time column (1, nS | 1) in
// all of them (odd for the flush, whose lanes read along c).  Portfolio risks on a 30x32 grid, 2^18
// paths, by row and by column: 992 and 530 us in FP32, 2240 and 1180 us in FP64.  With 8 banks (120x60)
// the two are within 1% of each other, with 16 (60x30) by row is 1-1.5% faster, so those stay by row.
struct NodeStride
{
    int l, c;
};
CF_HD NodeStride node_stride(int nS, int nT)
{
    NodeStride d;
    d.l = nT % 8 ? nT : 1;
    d.c = nT % 8 ? 1 : nS | 1;
    return d;
}
CF_HD int node_words(int nS, int nT) { return nT % 8 ? nS * nT : (nS | 1) * nT; }

struct alignas(16) FxVol  // of one step and interval: the slope as bh 2^32 + bl, bl signed
{
    long long a;
    int bl, bh;
};
struct alignas(32) FxStep  // the reverse's split of a step's vols over the time nodes (16-byte loads)
{
    long long tw;  // weight of column colB, units of 2^-62
    double sq;     // sqrt(dt)
    int atA, atB;    // time columns times node_stride().c: their places in the node slab
    int colA, colB;  // time columns
};

// Number of knots up to y (upper_bound): the state's interval.  x0h: high word of the first edge
// (edges are multiples of 2^32).
CF_HD int fx_interval(const long long* buckets, int nBuckets, int shift, int x0h, long long y)
{
    const int k = ((int)(y >> 32) - x0h) >> shift;
    const long long e = buckets[k < 0 ? 0 : k < nBuckets ? k : nBuckets - 1];
    return ((int)e & ((1 << FX_LO_BITS) - 1)) + (y >= e ? 1 : 0);
}

// sqrt(dt) sigma at y.
CF_HD long long fx_vol(long long a, int bl, int bh, long long y, long long center, int sh)
{
    const long long D = (long long)((unsigned long long)(y - center) << sh);
    const int dl = (int)(unsigned)D, dh = (int)((D - dl) >> 32);
    const long long mid = (long long)dh * bl + (long long)dl * bh + 0x80000000LL;
    return a + (long long)dh * bh + (mid >> 32);
}

// One log-Euler step: y + v (g - v / 2), rounded to the multiples of the unit grid = 2^k that a double
// log S has near log S0 (half: 2^31 grid).  The state has spare bits below that unit, but
// the reference rounds every step there, and a barrier's smoothing band amplifies such a rounding by
// barrier / band width: with its grid the golden barrier risks agree with the reference's to 1e-13 to
// 5e-13 of the largest, without to 4e-13 to 1.04e-12.
CF_HD long long fx_step(long long y, long long v, long long g, int r, long long half, long long grid)
{
    return fx_mul_add(v, g - (v >> (4 - r)), y, half) & -grid;
}

// 8 (1 - exp(-w)) in units of 2^-62, for 0 <= w < 1/32 in units of 2^-(57 - r): the series of
// (1 - exp(-w)) / w to the eighth order in u = 8 w (the ninth is below 2^-60).
constexpr int FX_SMOOTH_BITS = 5;
CF_HD long long fx_one_minus_exp8(long long w, int r)
{
    constexpr double one = 4611686018427387904.0;  // 2^62
    constexpr long long c[9] = {(long long)one,
                                (long long)(-one / 2 / 8),
                                (long long)(one / 6 / 64),
                                (long long)(-one / 24 / 512),
                                (long long)(one / 120 / 4096),
                                (long long)(-one / 720 / 32768),
                                (long long)(one / 5040 / 262144),
                                (long long)(-one / 40320 / 2097152),
                                (long long)(one / 362880 / 16777216)};
    const long long u = (long long)((unsigned long long)w << (10 + r));  // units of 2^-64, below 2^62
    long long s = c[8];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int k = 7; k >= 0; --k) s = fx_mul_add(s, u, c[k]);
    return fx_mul_add(s, u, 0);
}

// ---------------------------------------------------------------------------------------
// exp(a) for |a| < 16 in units of 2^-58, as m 2^(n - 61) with m of 62 bits (relative error below 2^-57):
// a log2(e) = n + i / 128 + z, |z| <= 2^-8; table[i] = 2^(i / 128) in units of 2^-61, 2^z - 1 a
// quintic in z.  A double exp takes a warp 321 cycles of its SM, this about 70.
// ---------------------------------------------------------------------------------------
constexpr int FX_EXP_BITS = 7, FX_A = 58;
CF_HD long long fx_exp(const long long* table, long long a, int& n)
{
    const long long t = fx_mul_add(a, 3326628274461080623LL, 1LL << 47);  // log2(e) 2^61; half of 2^-7 added
    n = (int)(t >> 55);
    const long long T = table[(int)(t >> 48) & ((1 << FX_EXP_BITS) - 1)];
    const long long v = ((t & ((1LL << 48) - 1)) - (1LL << 47)) * 32768;  // z in units of 2^-70
    // ln(2)^k / k! in units of 2^-58, 2^-52, ..., 2^-34
    long long s = fx_mul_add(22906878LL, v, 10575244791LL);
    s = fx_mul_add(s, v, 3905754423444LL);
    s = fx_mul_add(s, v, 1081884007225522LL);
    s = fx_mul_add(s, v, 199786072581291495LL);
    return fx_mul_add(fx_mul_add(s, v, 0), T, T);
}

// ---------------------------------------------------------------------------------------
// Inverse normal of a whole-number draw, to 2^-55.  up in [1, 2^31] counts from the nearer end of
// the generator's range.  Its leading bit and the next 9 select a piece, the 22 bits after them
// are the variable of a quartic: coefficients of order 0 to 2 in units of 2^-59, of order 3 and 4
// in 2^-55, the variable scaled to [0, 1/2).  Beasley-Springer-Moro changes formula at u = 0.08
// with a step of 1e-9, so the piece that holds the change exists twice: from brk upwards the
// index is one higher.  The value is the distance from zero, in units of 2^-59.  (A record is two
// 16-byte loads: the table reads are the path kernels' largest use of the L1 data path, and a
// sextic with 7 bits took three.)
// ---------------------------------------------------------------------------------------
constexpr int FXG_SUB_BITS = 9;
constexpr int FXG_PIECES = (32 << FXG_SUB_BITS) + 1;
struct alignas(32) FxgPiece
{
    long long c0, c1, c2;
    int c3, c4;
};

CF_HD int fxg_piece(unsigned up, unsigned brk, int& w)
{
#ifdef __CUDA_ARCH__
    const int lz = __clz((int)up);
#else
    const int lz = __builtin_clz(up);
#endif
    const unsigned nrm = up << lz;
    w = (int)((nrm << (FXG_SUB_BITS + 1)) >> 1);
    return ((31 - lz) << FXG_SUB_BITS) + (int)((nrm >> (31 - FXG_SUB_BITS)) & ((1u << FXG_SUB_BITS) - 1u)) + (up >= brk ? 1 : 0);
}

CF_HD long long fxg_value(const FxgPiece& c, int w)
{
#ifdef __CUDA_ARCH__
    const int q = __mulhi(c.c3 + __mulhi(c.c4, w), w);
#else
    const int q = (int)(((long long)(c.c3 + (int)(((long long)c.c4 * w) >> 32)) * w) >> 32);
#endif
    const long long s = c.c1 + fx_mul32(c.c2 + (long long)q * 16, w);
    return c.c0 + fx_mul32(s, w);
}

}  // namespace cf
