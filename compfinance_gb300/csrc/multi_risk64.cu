// FP64 AADriskMulti of a European portfolio on the Dupire model in fixed point: the stages of
// multi_risk32.cu (paths grouped by maturity and strike bucket, chunks of one bucket swept back into
// a shared slab) with the path arithmetic and the slab of dupire_fx64 (fixed64.h, fx_device.cuh).
//
// What bounds it: the reverse, one sweep per path and maturity it is in the money for, by the
// shared-memory adds and the dependent chain of the adjoint.  The former kernel (multi_kernel.cu,
// which keeps Black-Scholes and models beyond the fixed-point ranges) ran at the FP64 pipe's and the
// global 64-bit atomics' rates: each path-step of a maturity cost eight of them.  Measured, 200
// options on the 60x30 grid, 40 steps, 2^18 Sobol paths: 3.76 -> 1.12 ms (6.8 before its Gaussians
// and sums were cheapened).
#include <cuda_runtime.h>

#include "fx_device.cuh"
#include "multi32.h"
#include "occupancy.h"

namespace cf {

namespace {

constexpr int FB = 128;  // threads of a forward block

struct Fwd64
{
    size_t val, hist, bucket, ks, evOff, base, total;
};

__host__ __device__ inline Fwd64 fwd64_layout(int rng, const Multi32Args& A)
{
    Fwd64 L;
    size_t off = 0;
    auto take = [&](size_t n) {
        const size_t o = off;
        off += (n + 15) & ~size_t(15);
        return o;
    };
    L.val = take(size_t(A.nBuckets) * 16);  // sum of S per bucket
    L.hist = take(size_t(A.nBuckets) * 4);  // entries per bucket
    L.bucket = take(size_t(A.p.fx.nBuckets) * 8);
    L.ks = take(size_t(A.nKs) * 8);
    L.evOff = take(size_t(A.p.nEv + 1) * 4);
    L.base = take(rng == RNG_SOBOL ? size_t(FB / 32) * (size_t(A.p.nSteps) | 1) * 4 : 0);
    L.total = off;
    return L;
}

struct Rev64
{
    size_t node, inv, interval, bucket, spot, misc, total;
};

__host__ __device__ inline Rev64 rev64_layout(const Multi32Args& A)
{
    Rev64 L;
    size_t off = 0;
    auto take = [&](size_t n) {
        const size_t o = off;
        off += (n + 15) & ~size_t(15);
        return o;
    };
    L.node = take(size_t(node_words(A.p.nS, A.p.nT)) * 12);
    L.inv = take(size_t(A.p.nS + 1) * 8);
    L.interval = take(size_t(A.p.nS + 1) * 16);
    L.bucket = take(size_t(A.p.fx.nBuckets) * 8);
    L.spot = take(16);
    L.misc = take(16);
    L.total = off;
    return L;
}

__device__ __forceinline__ long long vol_at(const FxParams& f, const long long* sBucket, int pitch, int s, long long y,
                                            int& lo)
{
    lo = fx_interval(sBucket, f.nBuckets, f.shift, f.x0h, y);
    const int4 c = __ldg(reinterpret_cast<const int4*>(f.vol + s * pitch + lo));
    return fx_vol((long long)(((unsigned long long)(unsigned)c.y << 32) | (unsigned)c.x), c.z, c.w, y, f.center, f.sh);
}

template <int RNGK>
__global__ void __launch_bounds__(FB, 8) multi64_forward(const Multi32Args A)
{
    constexpr int NP = RNGK == RNG_MRG ? 2 : 1;
    const McParams& p = A.p;
    extern __shared__ __align__(128) unsigned char smem[];
    const Fwd64 L = fwd64_layout(RNGK, A);
    long long* sVal = reinterpret_cast<long long*>(smem + L.val);
    int* hist = reinterpret_cast<int*>(smem + L.hist);
    long long* sBucket = reinterpret_cast<long long*>(smem + L.bucket);
    long long* sKs = reinterpret_cast<long long*>(smem + L.ks);
    int* sEvOff = reinterpret_cast<int*>(smem + L.evOff);
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int nSteps = p.nSteps, nEv = p.nEv, nB = A.nBuckets, pitch = p.nS + 1;
    for (int i = tid; i < 2 * nB; i += FB) sVal[i] = 0;
    for (int i = tid; i < nB; i += FB) hist[i] = 0;
    for (int i = tid; i < p.fx.nBuckets; i += FB) sBucket[i] = p.fx.bucket[i];
    for (int i = tid; i < A.nKs; i += FB) sKs[i] = A.ksI[i];
    for (int i = tid; i <= nEv; i += FB) sEvOff[i] = A.evOff[i];
    __syncthreads();
    const double yUnit = ldexp(1.0, p.fx.r - FX_Y);
    const long long nPath = p.nPath;

    // maturity e of a path: bucket = number of sorted strikes below the spot
    auto event = [&](int e, long long path, long long y) {
        const int o = sEvOff[e] - e, n = sEvOff[e + 1] - sEvOff[e] - 1;
        int lo = 0, hi = n;
        while (lo < hi)
        {
            const int mid = (lo + hi) >> 1;
            if (y > sKs[o + mid]) lo = mid + 1;
            else hi = mid;
        }
        const size_t at = size_t(e) * size_t(nPath) + size_t(path);
        A.evB[at] = (unsigned short)lo;
        if (lo > 0)
        {
            const double S = exp(fma((double)y, yUnit, p.x0d));
            A.evS64[at] = S;
            const int bk = sEvOff[e] + lo;
            fix_add_s(sVal + 2 * bk, S);
            atomicAdd(hist + bk, 1);
        }
    };
    auto runUnit = [&](int nAct, long long path0, auto&& gen) {
        long long y[NP];
#pragma unroll
        for (int a = 0; a < NP; ++a) y[a] = 0;
        const int e0 = __ldg(p.evAtStep);
        if (e0 >= 0)
#pragma unroll
            for (int a = 0; a < NP; ++a)
                if (a < nAct) event(e0, path0 + a, 0);
        longlong2* rec = A.rec64 + size_t(path0) * nSteps;
        for (int s = 0; s < nSteps; ++s)
        {
            const long long g = gen(s);
#pragma unroll
            for (int a = 0; a < NP; ++a)
            {
                if (a >= nAct) break;
                const long long ga = a ? -g : g;
                rec[a * nSteps + s] = make_longlong2(y[a], ga);
                int lo;
                const long long v = vol_at(p.fx, sBucket, pitch, s, y[a], lo);
                y[a] = fx_step(y[a], v, ga, p.fx.r, p.fx.half, p.fx.grid);
            }
            const int e = __ldg(p.evAtStep + s + 1);
            if (e >= 0)
#pragma unroll
                for (int a = 0; a < NP; ++a)
                    if (a < nAct) event(e, path0 + a, y[a]);
        }
    };
    if (RNGK == RNG_MRG)
    {
        // rounds of FB consecutive pairs, claimed from the launch counter
        const long long nUnits = (nPath + 1) / 2, nRounds = (nUnits + FB - 1) / FB;
        __shared__ unsigned long long sRound;
        for (;;)
        {
            __syncthreads();
            if (tid == 0) sRound = atomicAdd(p.claim, 1ull);
            __syncthreads();
            const long long u = (long long)sRound * FB + tid;
            if ((long long)sRound >= nRounds) break;
            if (u >= nUnits) continue;
            MrgState st = mrg_jump(p.seed1, p.seed2, (unsigned long long)(p.firstPath / 2 + u) * nSteps, p.mrgJumpA,
                                   p.mrgJumpB);
            runUnit((2 * u + 1 < nPath) ? 2 : 1, 2 * u, [&](int) { return mrg_gauss_fx(p.fx, mrg_next(st)); });
        }
    }
    else
    {
        // a warp's batch b: lane l runs Sobol index n = 32 b + l (path n - 1)
        unsigned* base = reinterpret_cast<unsigned*>(smem + L.base) + wib * (nSteps | 1);
        const long long nBatches = nPath / 32 + 1;
        for (;;)
        {
            unsigned long long bc = 0;
            if (lane == 0) bc = atomicAdd(p.claim, 1ull);
            const long long b = (long long)__shfl_sync(0xffffffffu, bc, 0);
            if (b >= nBatches) break;
            __syncwarp();
            for (int d = lane; d < nSteps; d += 32)
                base[d] = sobol_state(p.sobolDir, nSteps, d, (unsigned long long)(p.firstPath + b * 32));
            __syncwarp();
            const long long n = b * 32 + lane;
            if (n >= 1 && n <= nPath)
                runUnit(1, n - 1, [&](int i) {
                    return sobol_gauss_fx(p.fx, base[i] ^ sobol_low(p, i, lane));
                });
        }
    }
    __syncthreads();
    for (int i = tid; i < nB; i += FB) fix_flush(&A.accVal[2 * (5 * i + 1)], &sVal[2 * i]);
    for (int i = tid; i < nB; i += FB)
        if (hist[i]) atomicAdd(A.cnt + i, hist[i]);
}

// At least three blocks of 256 threads per SM asked of the compiler, which uses 64 registers: four fit.  The
// 60x30 grid's slab takes 22 KB, the 120x60 grid's 86 KB (two blocks).
__global__ void __launch_bounds__(M64_BLOCK, 3) multi64_reverse(const Multi32Args A)
{
    const McParams& p = A.p;
    extern __shared__ __align__(128) unsigned char smem[];
    const Rev64 L = rev64_layout(A);
    unsigned* node = reinterpret_cast<unsigned*>(smem + L.node);
    long long* sInv = reinterpret_cast<long long*>(smem + L.inv);
    FxInterval* sIv = reinterpret_cast<FxInterval*>(smem + L.interval);
    long long* sBucket = reinterpret_cast<long long*>(smem + L.bucket);
    long long* spotSlab = reinterpret_cast<long long*>(smem + L.spot);
    int* misc = reinterpret_cast<int*>(smem + L.misc);
    const int tid = threadIdx.x;
    const int nS = p.nS, nSteps = p.nSteps, nNodes = node_words(nS, p.nT), nB = A.nBuckets, pitch = nS + 1;
    for (int i = tid; i < 3 * nNodes; i += M64_BLOCK) node[i] = 0;
    for (int i = tid; i < nS + 1; i += M64_BLOCK)
    {
        sIv[i] = p.fx.interval[i];
        sInv[i] = p.fx.inv[i];
    }
    for (int i = tid; i < p.fx.nBuckets; i += M64_BLOCK) sBucket[i] = p.fx.bucket[i];
    if (tid < 2) spotSlab[tid] = 0;
    __syncthreads();
    const int nChunks = __ldg(A.chunkStart + nB), r = p.fx.r;
    for (;;)
    {
        if (tid == 0) misc[0] = atomicAdd(A.work, 1);
        __syncthreads();
        // the last maturities, whose sweeps are the longest, first
        const int c = nChunks - 1 - misc[0];
        if (c < 0) break;
        // bucket of chunk c: the last b with chunkStart[b] <= c (empty buckets share starts)
        int lo = 0, hi = nB;
        while (hi - lo > 1)
        {
            const int mid = (lo + hi) >> 1;
            if (__ldg(A.chunkStart + mid) <= c) lo = mid;
            else hi = mid;
        }
        const int b = lo;
        int e0 = 0, e1 = p.nEv;  // maturity of bucket b: the last e with evOff[e] <= b
        while (e1 - e0 > 1)
        {
            const int mid = (e0 + e1) >> 1;
            if (__ldg(A.evOff + mid) <= b) e0 = mid;
            else e1 = mid;
        }
        const int iE = __ldg(p.evPoint + e0);
        const int first = __ldg(A.start + b) + (c - __ldg(A.chunkStart + b)) * M32_CHUNK;
        const int end = __ldg(A.start + b + 1);
        const int count = end - first < M32_CHUNK ? end - first : M32_CHUNK;
        long long* row = A.accRisk + 2 * size_t(b) * A.nParam;
        if (tid < count)
        {
            const longlong2 e = A.list64[first + tid];
            // d payoff / d x_e = S_e, carried in the Gaussians' unit
            double ax = __longlong_as_double(e.y) * 0x1p-59;
            const longlong2* rr = A.rec64 + size_t(e.x) * nSteps;
            longlong2 next = iE > 0 ? __ldg(rr + iE - 1) : make_longlong2(0, 0);
            for (int s = iE - 1; s >= 0; --s)
            {
                const longlong2 cur = next;
                if (s > 0) next = __ldg(rr + s - 1);
                int k;
                const long long v = vol_at(p.fx, sBucket, pitch, s, cur.x, k);
                const double av = ax * (double)(cur.y - 2 * (v >> (4 - r)));  // d x_{s+1} / d v = g - v
                ax = fma(av, __ldg(p.fx.slope + s * pitch + k), ax);
                if (av != 0.0) fx_vol_adjoint(p, row, node, nNodes, sIv, sInv, s, k, cur.x, av);
            }
            fix_add_s(spotSlab, ax * 0x1p59 / p.spot);  // x_0 = log(spot)
        }
        __syncthreads();
        fx_node_flush<true>(p, row, node, nNodes, M64_BLOCK);
        if (tid == 0)
        {
            fix_flush(row, spotSlab);
            spotSlab[0] = spotSlab[1] = 0;
        }
        __syncthreads();
    }
}

const void* fwd_ptr(int rng)
{
    return rng == RNG_MRG ? (const void*)&multi64_forward<RNG_MRG> : (const void*)&multi64_forward<RNG_SOBOL>;
}

}  // namespace

size_t m64_forward_smem(int rng, const Multi32Args& a) { return fwd64_layout(rng, a).total; }
size_t m64_reverse_smem(const Multi32Args& a) { return rev64_layout(a).total; }

int m64_occupancy(int rng, size_t smemFwd, size_t smemRev, int* occFwd, int* occRev)
{
    const int e = kernel_occupancy(fwd_ptr(rng), FB, smemFwd, occFwd);
    return e ? e : kernel_occupancy((const void*)&multi64_reverse, M64_BLOCK, smemRev, occRev);
}

int launch_multi64(int rng, int gridFwd, size_t smemFwd, int gridRev, size_t smemRev, const Multi32Args& a,
                   void* stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    Multi32Args q = a;
    void* args[] = {&q};
    cudaError_t e = cudaLaunchKernel(fwd_ptr(rng), dim3(gridFwd), dim3(FB), args, smemFwd, st);
    if (!e) e = (cudaError_t)launch_multi32_scan(a, stream);
    if (!e) e = (cudaError_t)launch_multi32_scatter(a, true, stream);
    if (!e) e = cudaLaunchKernel((const void*)&multi64_reverse, dim3(gridRev), dim3(M64_BLOCK), args, smemRev, st);
    return (int)e;
}

}  // namespace cf
