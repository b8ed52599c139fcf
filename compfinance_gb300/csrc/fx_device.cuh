// Reverse step of the fixed-point Dupire kernels (mc_dupire_fx64.cuh, multi_risk64.cu): the adjoint of
// one step's vol into a slab of 96-bit words of the local-vol nodes in shared memory, in units of
// 2^-60, held as three arrays of 32-bit words [3][nNodes], each laid out by node_stride().
#pragma once
#include "cf_device.cuh"

namespace cf {

// v[k] 2^sft, rounded, into words at[k], k < n (2 or 4).  Of each word the low two 32-bit adds return
// their old values for the carries; the third is rarely needed (a negative value's sign word nearly
// always meets a carry).  The adds of one kind are issued together: one after the other, each with
// its carry, four words cost eight round trips to shared memory instead of two.
__device__ __forceinline__ void fx_node_add(unsigned* node, int nNodes, const int (&at)[4], long long (&v)[4], int n, int sft)
{
    unsigned a1[4], a2[4], o[4];
    if (sft < 0)
    {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = sft < -62 ? 0 : (v[k] + (1LL << (-sft - 1))) >> -sft;
        sft = 0;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < 2 || n > 2) o[k] = atomicAdd(node + at[k], (unsigned)v[k] << sft);
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        const unsigned l = (unsigned)v[k], h = (unsigned)((unsigned long long)v[k] >> 32), a0 = l << sft;
        const unsigned c = o[k] + a0 < o[k] ? 1u : 0u, b1 = __funnelshift_l(l, h, sft);
        a1[k] = b1 + c;
        a2[k] = (unsigned)((int)h >> (sft ? 32 - sft : 31)) + (a1[k] < c ? 1u : 0u);  // b1 + c may wrap to 0
        if (k < 2 || n > 2) o[k] = atomicAdd(node + nNodes + at[k], a1[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        a2[k] += o[k] + a1[k] < o[k] ? 1u : 0u;
        if (a2[k] && (k < 2 || n > 2)) atomicAdd(node + 2 * nNodes + at[k], a2[k]);
    }
}

// Adjoint av of the vol sqrt(dt) sigma of step s at state y in interval lo, split over the interval's
// two knots and the step's two time columns; beyond the slab's range (p.fx.nodeShift) straight into
// the accumulator pairs acc[1 + node].
__device__ __forceinline__ void fx_vol_adjoint(const McParams& p, long long* acc, unsigned* node, int nNodes,
                                               const FxInterval* sIv, const long long* sInv, int s, int lo, long long y,
                                               double av)
{
    const int nS = p.nS, dl = p.fx.node.l;
    const FxInterval iv = sIv[lo];
    const bool inner = lo > 0 && lo < nS;  // two knots; one at the flat ends
    // weight of the upper knot, units of 2^-59
    const long long t = inner ? fx_mul_add(sInv[lo], (long long)((unsigned long long)(y - iv.x) << iv.sh), 0) : 0;
    const int jl = lo - (lo > 0 ? 1 : 0);
    const longlong2 s0 = __ldg(reinterpret_cast<const longlong2*>(p.fx.step + s));
    const int2 at2 = __ldg(reinterpret_cast<const int2*>(&p.fx.step[s].atA));
    // the adjoint of sigma as N 2^sft units of 2^-60: its 53-bit mantissa
    const double c = av * __longlong_as_double(s0.y);
    const int hi = __double2hiint(c), E = (hi >> 20) & 0x7ff;
    const int sft = E - (1023 - FIX_LO_SHIFT + 52);
    if (sft <= p.fx.nodeShift)
    {
        const unsigned long long m =
            ((unsigned long long)(unsigned)((hi & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(c);
        const long long N = hi < 0 ? -(long long)m : (long long)m;
        const long long nR = fx_mul_add(N * 32, t, 0), nL = N - nR;
        const long long rB = fx_mul_add(nR * 4, s0.x, 0), lB = fx_mul_add(nL * 4, s0.x, 0);
        const int at[4] = {jl * dl + at2.x, jl * dl + at2.y, (jl + 1) * dl + at2.x, (jl + 1) * dl + at2.y};
        long long v[4] = {nL - lB, lB, nR - rB, rB};
        fx_node_add(node, nNodes, at, v, inner ? 4 : 2, sft);
    }
    else
    {
        const double cR = c * ((double)t * 0x1p-59), cL = c - cR;
        const double tw = (double)s0.x * 0x1p-62;
        const int nT = p.nT;
        const int2 col = __ldg(reinterpret_cast<const int2*>(&p.fx.step[s].colA));
        acc += 2 * (1 + jl * nT);
        fix_add(acc + 2 * col.x, cL - cL * tw);
        fix_add(acc + 2 * col.y, cL * tw);
        if (inner)
        {
            fix_add(acc + 2 * (nT + col.x), cR - cR * tw);
            fix_add(acc + 2 * (nT + col.y), cR * tw);
        }
    }
}

// Whole block (threads of them): the slab into the accumulator pairs acc[1 + node], and cleared.
// STRIDED: the slab may be by time column (p.fx.node); without it the loop is by row alone, whose
// second copy made a barrier's sweep 2% slower.
template <bool STRIDED>
__device__ __forceinline__ void fx_node_flush(const McParams& p, long long* acc, unsigned* node, int nNodes, int threads)
{
    const int nS = p.nS, nT = p.nT;
    auto flush = [&](int i, int k) {
        const unsigned n0 = node[k], n1 = node[k + nNodes], n2 = node[k + 2 * nNodes];
        if (n0 | n1 | n2)
        {
            node[k] = node[k + nNodes] = node[k + 2 * nNodes] = 0;
            long long hi, lo;
            fix_split_slab(n0, n1, n2, hi, lo);
            long long* at = acc + 2 * (1 + i);
            if (hi) atomicAdd(reinterpret_cast<unsigned long long*>(at), (unsigned long long)hi);
            if (lo) atomicAdd(reinterpret_cast<unsigned long long*>(at + 1), (unsigned long long)lo);
        }
    };
    if (!STRIDED || p.fx.node.c == 1)
        for (int i = threadIdx.x; i < nS * nT; i += threads) flush(i, i);
    else
        for (int l = threadIdx.x >> 5; l < nS; l += threads >> 5)
            for (int c = threadIdx.x & 31; c < nT; c += 32) flush(l * nT + c, l * p.fx.node.l + c * p.fx.node.c);
}

}  // namespace cf
