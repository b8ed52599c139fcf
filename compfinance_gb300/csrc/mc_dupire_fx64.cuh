// FP64 form of the Dupire value and risk runs (European and smoothed up-and-out products:
// mcSimul and mcSimulAAD, mcBase.h:267-308, 427-532; mcMdlDupire.h:238-280; mcPrd.h:113-288), with
// the path arithmetic in 64-bit fixed point (fixed64.h).
//
// What bounds it: the generic kernel keeps GB300's FP64 pipe 83% busy (16 cycles per warp and
// operation, about 110 operations per path-step: both branches of the inverse normal, the interval
// search, the splits of the sums).  In fixed point a path-step takes no FP64 operation: the inverse
// normal is a quartic of the integer draw (two 64 x 32-bit products), the interval one bucket
// lookup and comparison, the vol and the step one rounded 64 x 64-bit product each.  States have
// the unit of a double near log S0 (fx_step), vols 61 fraction bits, Gaussians 59.  Doubles remain where
// magnitudes range widely: payoffs, exp at maturity, and the reverse's adjoint, whose products with
// the vol weights are again whole numbers.  Measured (60x30 weekly barrier, mrg32k3a): risk 9.5 ->
// 0.59 ms at 2^18 paths and 141 -> 5.6 ms at 2^22, value 5.2 -> 0.30 ms at 2^18; 141 instructions per
// path-step of the value run (ncu), issue 58%, ALU pipe 54%, L1 data path 43% of their peaks.
//
// Rounds, compaction of the paths with an adjoint and the claimed chunks follow dupire_risk32:
// a block runs rounds of RB units, lists the paths whose adjoint seed is not zero, and sweeps RB of
// them at a time back from maturity.  The sweep recomputes each step's interval and vol from the
// stored state.  The adjoint of a vol is split over two knots and two time columns by rounded integer
// products of its 53-bit mantissa, which are added to a slab of 96-bit words in shared memory, in
// units of 2^-60 (two 32-bit adds each, rarely three).  After each sweep the slab goes to the accumulators.  All sums
// are of whole numbers rounded per contribution, so results do not depend on the grid.
#pragma once
#include <cuda_runtime.h>

#include "fx_device.cuh"

namespace cf {

namespace {

struct FxLayout
{
    size_t slab, node, inv, interval, bucket, list, cnt, base, total;
};

// pending paths: fewer than three blocks of them, in a ring of a power of two
__host__ __device__ constexpr int fx_list(int block) { return block <= 128 ? 512 : 2048; }

__host__ __device__ inline FxLayout fx_layout(int rng, int block, const McParams& p)
{
    FxLayout L;
    size_t off = 0;
    auto take = [&](size_t n) {
        const size_t o = off;
        off += (n + 15) & ~size_t(15);
        return o;
    };
    const bool risk = p.nRisk > 0;
    L.slab = take(size_t(4 + 2 * p.nPay + 2) * 16);
    L.node = take(risk ? size_t(p.nS) * p.nT * 12 : 0);  // local-vol nodes of the current sweep
    L.inv = take(risk ? size_t(p.nS + 1) * 8 : 0);
    L.interval = take(risk ? size_t(p.nS + 1) * 16 : 0);
    L.bucket = take(size_t(p.fx.nBuckets) * 8);
    L.list = take(risk ? size_t(fx_list(block)) * 4 : 0);
    L.cnt = take(size_t(block / 32) * 4 + 16);        // claimed chunk, per-warp counts
    L.base = take(rng == RNG_SOBOL ? size_t(block / 32) * (size_t(p.nSteps) | 1) * 4 : 0);
    L.total = off;
    return L;
}

// Resident blocks asked of the compiler: 7 x 128 or 2 x 384 threads (72 and 80 registers) for risk; at 72 the
// barrier spills 44 bytes with mrg32k3a and 24 with Sobol, the European 28 with mrg32k3a.  The large block
// shares the slab of a 120 x 60 grid (86 KB), of which two fit an SM.
template <int PROD, int RNGK, bool RISK, int RB>
__global__ void __launch_bounds__(RB, RISK ? (RB == 128 ? 7 : 2) : 8) dupire_fx64(const McParams p)
{
    constexpr int NP = RNGK == RNG_MRG ? 2 : 1;
    constexpr bool UOC = PROD == PROD_UOC;
    constexpr int LIST = fx_list(RB), RW = RB / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    const FxLayout L = fx_layout(RNGK, RB, p);
    long long* slab = reinterpret_cast<long long*>(smem + L.slab);  // [0,2) spot adjoint, payoffs from 8
    long long* paySlab = slab + 8;
    unsigned* node = reinterpret_cast<unsigned*>(smem + L.node);  // [3][nNodes]
    long long* sInv = reinterpret_cast<long long*>(smem + L.inv);
    FxInterval* sIv = reinterpret_cast<FxInterval*>(smem + L.interval);
    long long* sBucket = reinterpret_cast<long long*>(smem + L.bucket);
    unsigned* list = reinterpret_cast<unsigned*>(smem + L.list);
    long long* sClaim = reinterpret_cast<long long*>(smem + L.cnt);
    int* cnt = reinterpret_cast<int*>(smem + L.cnt + 16);
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int nS = p.nS, nT = p.nT, nSteps = p.nSteps, nPay = p.nPay, nNodes = RISK ? nS * nT : 0;
    for (int i = tid; i < 2 * (4 + 2 * nPay + 2); i += RB) slab[i] = 0;
    for (int i = tid; i < 3 * nNodes; i += RB) node[i] = 0;
    if (RISK)
        for (int i = tid; i < nS + 1; i += RB)
        {
            sIv[i] = p.fx.interval[i];
            sInv[i] = p.fx.inv[i];
        }
    for (int i = tid; i < p.fx.nBuckets; i += RB) sBucket[i] = p.fx.bucket[i];
    __syncthreads();

    const int r = p.fx.r, nBuckets = p.fx.nBuckets, bShift = p.fx.shift, x0h = p.fx.x0h, dShift = p.fx.sh;
    const long long center = p.fx.center, half = p.fx.half, grid = p.fx.grid, yTop = p.fx.yTop, yBand = p.fx.yBand;
    const FxVol* vols = p.fx.vol;
    const int pitch = nS + 1;
    const double yUnit = ldexp(1.0, r - FX_Y);
    const double w0 = nPay > 0 && RISK ? p.w[0] : 0.0, w1 = nPay > 1 && RISK ? p.w[1] : 0.0;
    const bool evEvery = p.evEvery != 0;

    // log S = log S0 + y is a double (the state has its grid)
    auto spotOf = [&](long long y) { return exp(fma((double)y, yUnit, p.x0d)); };
    // survival factor of a date in the band, (barSmooth - S) / twoSmooth, and its spot
    auto bandFactor = [&](long long y, double& S) -> double {
        if (p.fx.bandScale > 0.0)
        {
            const double f = (double)fx_one_minus_exp8(yTop - y, r) * p.fx.bandScale;
            S = fma(-p.twoSmooth, f, p.barSmooth);
            return f;
        }
        S = spotOf(y);
        return (p.barSmooth - S) / p.twoSmooth;
    };
    auto volAt = [&](int s, long long y, int& lo) -> long long {
        lo = fx_interval(sBucket, nBuckets, bShift, x0h, y);
        const int4 c = __ldg(reinterpret_cast<const int4*>(vols + s * pitch + lo));
        return fx_vol((long long)(((unsigned long long)(unsigned)c.y << 32) | (unsigned)c.x), c.z, c.w, y, center, dShift);
    };
    // scratch [ring slot][field][point][thread] of 64-bit words, 32-bit offsets: the Gaussian, the
    // state per path and, for the barrier, the survival factor before band dates per path.  Point
    // nSteps holds the adjoint seeds of the state and of the survival factor.
    const int Ti = int(gridDim.x) * RB;
    const int rowStride = (nSteps + 1) * Ti;
    constexpr int F_G = 0, F_Y = 1, F_B = 1 + NP, NF = UOC ? 1 + 2 * NP : 1 + NP;
    const int slotStride = NF * rowStride;
    long long* const scr = reinterpret_cast<long long*>(p.scratch);
    long long* fs = scr;  // the slot of the current unit round
    const int myCol = int(blockIdx.x) * RB + tid;
    const int seedRow = nSteps * Ti;
    const double invTwo = -1.0 / p.twoSmooth;


    // ---------------------------------------------------------------------------------
    // One unit: forward, payoff sums, adjoint seeds; live[] says which paths have one.
    // ---------------------------------------------------------------------------------
    bool live[NP];
    auto forward = [&](int nAct, long long path0, auto&& gen) {
        long long y[NP];
        double alive[NP], bLast[NP], sT[NP];
        bool dead[NP], band[NP];
#pragma unroll
        for (int a = 0; a < NP; ++a)
        {
            y[a] = 0;
            alive[a] = 1.0;
            bLast[a] = sT[a] = 0.0;
            dead[a] = band[a] = live[a] = false;
        }
        if (!nAct) return;
        // product date at point i (for i < nSteps only the barrier's monitoring, above the band's start)
        auto event = [&](int i, int a) {
            const bool last = i == nSteps;
            if (UOC && !dead[a] && y[a] > yBand)
            {
                if (y[a] > yTop) dead[a] = true;
                else
                {
                    if (last)
                    {
                        bLast[a] = alive[a];
                        band[a] = true;
                    }
                    else if (RISK) fs[(F_B + a) * rowStride + i * Ti + myCol] = __double_as_longlong(alive[a]);
                    double S;
                    alive[a] *= bandFactor(y[a], S);
                }
            }
            if (last) sT[a] = spotOf(y[a]);
        };
        if (p.evAtStep[0] >= 0)
#pragma unroll
            for (int a = 0; a < NP; ++a)
                if (a < nAct) event(0, a);
        long long* pw = fs + myCol;
        for (int s = 0; s < nSteps; ++s, pw += Ti)
        {
            const long long g = gen(s);
            if (RISK) __stcs(pw, g);
#pragma unroll
            for (int a = 0; a < NP; ++a)
            {
                if (a >= nAct) break;
                if (RISK) __stcs(pw + (F_Y + a) * rowStride, y[a]);
                int lo;
                const long long v = volAt(s, y[a], lo);
                y[a] = fx_step(y[a], v, a ? -g : g, r, half, grid);
            }
            const long long top = NP == 2 && y[NP - 1] > y[0] ? y[NP - 1] : y[0];
            if (s + 1 == nSteps || (UOC && top > yBand && (evEvery || __ldg(p.evAtStep + s + 1) >= 0)))
#pragma unroll
                for (int a = 0; a < NP; ++a)
                    if (a < nAct) event(s + 1, a);
        }
#pragma unroll
        for (int a = 0; a < NP; ++a)
        {
            if (a >= nAct) break;
            const double m = UOC && p.callPut ? p.strike - sT[a] : sT[a] - p.strike;
            const double euro = m > 0.0 ? m : 0.0;
            const double p0 = UOC ? (dead[a] ? 0.0 : alive[a] * euro) : euro;
            fix_add_s(&paySlab[0], p0);
            fix_add_s(&paySlab[2 * nPay], p0 * p0);
            if (UOC)
            {
                fix_add_s(&paySlab[2], euro);
                fix_add_s(&paySlab[2 * (nPay + 1)], euro * euro);
            }
            if (!RISK)
            {
                if (p.pathOut)
                {
                    p.pathOut[(path0 + a) * nPay] = p0;
                    if (UOC) p.pathOut[(path0 + a) * nPay + 1] = euro;
                }
                continue;
            }
            const double agg = UOC ? w0 * p0 + w1 * euro : w0 * p0;
            fix_add_s(&paySlab[2 * (2 * nPay)], agg);
            fix_add_s(&paySlab[2 * (2 * nPay + 1)], agg * agg);
            const double aEuro = !UOC ? w0 : dead[a] ? w1 : w0 * alive[a] + w1;
            double aAl = !UOC || dead[a] ? 0.0 : w0 * euro;
            double aF = m > 0.0 ? (UOC && p.callPut ? -aEuro : aEuro) : 0.0;
            if (band[a])
            {
                aF += aAl * bLast[a] * invTwo;
                double S;
                aAl *= bandFactor(y[a], S);
            }
            const double ax = aF * sT[a];
            live[a] = ax != 0.0 || aAl != 0.0;
            if (live[a])
            {
                fs[(F_Y + a) * rowStride + seedRow + myCol] = __double_as_longlong(ax);
                if (UOC) fs[(F_B + a) * rowStride + seedRow + myCol] = __double_as_longlong(aAl);
            }
        }
    };

    // Pending paths, first in first out: head, q2 and q1 are uniform over the block (q2 entries of
    // the round before last, then q1 of the last one; fewer than RB at the start of a round).
    int head = 0, q2 = 0, q1 = 0;
    auto collect = [&](int slot) -> int {
        const unsigned b0 = __ballot_sync(0xffffffffu, live[0]);
        const unsigned b1 = NP == 2 ? __ballot_sync(0xffffffffu, live[NP - 1]) : 0u;
        if (lane == 0) cnt[wib] = __popc(b0) + __popc(b1);
        __syncthreads();
        int total = 0, off = head + q2 + q1;
        for (int w = 0; w < RW; ++w)
        {
            off += w < wib ? cnt[w] : 0;
            total += cnt[w];
        }
        const unsigned lt = (1u << lane) - 1u, e = unsigned(slot) * (2 * RB) + 2 * tid;
        if (live[0]) list[(off + __popc(b0 & lt)) & (LIST - 1)] = e;
        if (NP == 2 && live[NP - 1]) list[(off + __popc(b0) + __popc(b1 & lt)) & (LIST - 1)] = e + 1;
        __syncthreads();
        return total;
    };

    auto sweep = [&](int n) {
        if (tid < n)
        {
            const unsigned e = list[(head + tid) & (LIST - 1)];
            const int a = int(e & 1);
            const long long* es = scr + int(e / (2 * RB)) * slotStride + int(blockIdx.x) * RB + int(e / 2 % RB);
            const long long* ey = es + (F_Y + a) * rowStride;
            const long long* eb = es + (F_B + a) * rowStride;
            double ax = __longlong_as_double(ey[seedRow]);
            double aAl = UOC ? __longlong_as_double(eb[seedRow]) : 0.0;
            ax *= 0x1p-59;  // carried in the Gaussians' unit
            // states and Gaussians are loaded three steps ahead (they come from DRAM), the vol and the slope of
            // a step one step ahead of its adds
            long long yA = __ldcs(ey + (nSteps - 1) * Ti), gA = __ldcs(es + (nSteps - 1) * Ti), yB = 0, gB = 0, yC = 0, gC = 0;
            if (nSteps >= 2)
            {
                yB = __ldcs(ey + (nSteps - 2) * Ti);
                gB = __ldcs(es + (nSteps - 2) * Ti);
            }
            if (nSteps >= 3)
            {
                yC = __ldcs(ey + (nSteps - 3) * Ti);
                gC = __ldcs(es + (nSteps - 3) * Ti);
            }
            int lo = fx_interval(sBucket, nBuckets, bShift, x0h, yA);
            int4 vc = __ldg(reinterpret_cast<const int4*>(vols + (nSteps - 1) * pitch + lo));
            double slope = __ldg(p.fx.slope + (nSteps - 1) * pitch + lo);
            for (int s = nSteps - 1; s >= 0; --s)
            {
                const long long y = yA, g = a ? -gA : gA;
                const long long v = fx_vol((long long)(((unsigned long long)(unsigned)vc.y << 32) | (unsigned)vc.x), vc.z, vc.w,
                                           y, center, dShift);
                const double av = ax * (double)(g - 2 * (v >> (4 - r)));  // d y_{s+1} / d v = g - v
                ax = fma(av, slope, ax);
                const int k = lo;
                yA = yB;
                gA = gB;
                yB = yC;
                gB = gC;
                if (s >= 3)
                {
                    yC = __ldcs(ey + (s - 3) * Ti);
                    gC = __ldcs(es + (s - 3) * Ti);
                }
                if (s >= 1)
                {
                    lo = fx_interval(sBucket, nBuckets, bShift, x0h, yA);
                    vc = __ldg(reinterpret_cast<const int4*>(vols + (s - 1) * pitch + lo));
                    slope = __ldg(p.fx.slope + (s - 1) * pitch + lo);
                }
                if (av != 0.0) fx_vol_adjoint(p, p.acc, node, nNodes, sIv, sInv, s, k, y, av);
                // the date at point s: survival below the barrier's smoothing band
                if (UOC && y > yBand && aAl != 0.0 && (evEvery ? s > 0 || p.evAtStep[0] >= 0 : __ldg(p.evAtStep + s) >= 0))
                {
                    double S;
                    const double f = bandFactor(y, S), before = __longlong_as_double(eb[s * Ti]);
                    ax += aAl * before * invTwo * S * 0x1p-59;
                    aAl *= f;
                }
            }
            fix_add_s(&slab[0], ax * 0x1p59 / p.spot);  // x_0 = log(spot)
        }
        head += n;
        __syncthreads();
        fx_node_flush<false>(p, p.acc, node, nNodes, RB);
        __syncthreads();
    };

    // End of a round (its paths in ring slot `slot`; slot < 0: after the last round): full sweeps,
    // and a partial one when paths of the round before last are pending (the next round rewrites
    // their slot) or no round follows.  Uniform over the block.
    auto endRound = [&](int slot) {
        const int count = q2 + q1 + (slot >= 0 ? collect(slot) : 0);
        int done = 0;
        for (;;)
        {
            const int left = count - done;
            const int n = left >= RB ? RB : (done < q2 || slot < 0) ? left : 0;
            if (n == 0) break;
            sweep(n);
            done += n;
        }
        const int old = q2 + q1 - done;
        q2 = old > 0 ? old : 0;
        q1 = count - done - q2;
    };

    long long it = 0;  // rounds this block has run: round it uses ring slot it mod R32_RING
    const long long cap = RISK && p.roundCap > 0 ? p.roundCap : LLONG_MAX;
    auto claim = [&](long long nRounds) {
        __syncthreads();  // every thread has read the previous chunk
        if (tid == 0)
        {
            const long long seen = (long long)*reinterpret_cast<volatile unsigned long long*>(p.claim);
            long long g = (nRounds - seen) / (2LL * gridDim.x);
            g = g > 1 ? g : 1;
            g = g < cap - it ? g : cap - it;
            sClaim[1] = g;
            sClaim[0] = g > 0 ? (long long)atomicAdd(p.claim, (unsigned long long)g) : LLONG_MAX;
        }
        __syncthreads();
    };
    auto slotOf = [&](long long i) {
        const int k = int(i % R32_RING);
        fs = scr + k * slotStride;
        return k;
    };
    if (RNGK == RNG_MRG)
    {
        const long long nUnits = (p.nPath + 1) / 2;
        const long long nRounds = (nUnits + RB - 1) / RB;
        for (;;)
        {
            claim(nRounds);
            const long long r0 = sClaim[0], G = sClaim[1];
            if (r0 >= nRounds) break;
            const long long u0 = r0 * RB + tid * G;
            MrgState st{};
            if (u0 < nUnits) st = mrg_jump(p.seed1, p.seed2, (unsigned long long)(p.firstPath / 2 + u0) * nSteps, p.mrgJumpA, p.mrgJumpB);
            for (long long j = 0; j < G; ++j, ++it)
            {
                const long long u = u0 + j;
                const int nAct = u < nUnits ? ((2 * u + 1 < p.nPath) ? 2 : 1) : 0;
                const int slot = RISK ? slotOf(it) : 0;
                forward(nAct, 2 * u, [&](int) { return mrg_gauss_fx(p.fx, mrg_next(st)); });
                if (RISK) endRound(slot);
            }
        }
    }
    else
    {
        const int bp = nSteps | 1;
        unsigned* base = reinterpret_cast<unsigned*>(smem + L.base) + wib * bp;
        const long long nBatches = p.nPath / 32 + 1;
        const long long nRounds = (nBatches + RW - 1) / RW;
        for (;;)
        {
            claim(nRounds);
            const long long r0 = sClaim[0], G = sClaim[1];
            if (r0 >= nRounds) break;
            for (long long j = 0; j < G; ++j, ++it)
            {
                const long long b = (r0 + j) * RW + wib, n = b * 32 + lane;
                int nAct = 0;
                if (b < nBatches)
                {
                    __syncwarp();
                    for (int d = lane; d < nSteps; d += 32)
                        base[d] = sobol_state(p.sobolDir, nSteps, d, (unsigned long long)(p.firstPath + b * 32));
                    __syncwarp();
                    nAct = (n >= 1 && n <= p.nPath) ? 1 : 0;
                }
                const int slot = RISK ? slotOf(it) : 0;
                forward(nAct, n - 1, [&](int i) {
                    return sobol_gauss_fx(p.fx, base[i] ^ sobol_low(p, i, lane));
                });
                if (RISK) endRound(slot);
            }
        }
    }
    if (RISK) endRound(-1);  // the paths still pending after the last round

    __syncthreads();
    if (RISK && tid == 0) fix_flush(&p.acc[0], &slab[0]);
    for (int i = tid; i < 2 * nPay + (RISK ? 2 : 0); i += RB) fix_flush(&p.acc[2 * (p.nRisk + i)], &paySlab[2 * i]);
    results_out(p);
}

}  // namespace

}  // namespace cf
