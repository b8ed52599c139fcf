// Reverse step of the fixed-point Dupire kernels (mc_dupire_fx64.cuh, multi_risk64.cu): the adjoint of
// one step's vol into a slab of 96-bit words of the local-vol nodes in shared memory, in units of
// 2^-60, held as three arrays of 32-bit words [3][nNodes].
#pragma once
#include "cf_device.cuh"

namespace cf {

// v 2^sft, rounded, into word i: the low two 32-bit adds return their old values for the carries; the
// third is rarely needed (a negative value's sign word nearly always meets a carry).
__device__ __forceinline__ void fx_node_add(unsigned* node, int nNodes, int i, long long v, int sft)
{
    if (sft < 0)
    {
        v = sft < -62 ? 0 : (v + (1LL << (-sft - 1))) >> -sft;
        sft = 0;
    }
    const unsigned l = (unsigned)v, h = (unsigned)((unsigned long long)v >> 32);
    const unsigned a0 = l << sft, a1 = __funnelshift_l(l, h, sft);
    unsigned a2 = (unsigned)((int)h >> (sft ? 32 - sft : 31));
    unsigned* at = node + i;
    const unsigned o0 = atomicAdd(at, a0), c0 = o0 + a0 < o0 ? 1u : 0u;
    const unsigned o1 = atomicAdd(at + nNodes, a1 + c0);
    // a1 + c0 wraps to 0 only with a carry of its own
    a2 += (a1 + c0 < c0 ? 1u : 0u) + (o1 + (a1 + c0) < o1 ? 1u : 0u);
    if (a2) atomicAdd(at + 2 * nNodes, a2);
}

// Adjoint av of the vol sqrt(dt) sigma of step s at state y in interval lo, split over the interval's
// two knots and the step's two time columns; beyond the slab's range (p.fx.nodeShift) straight into
// the accumulator pairs acc[1 + node].
__device__ __forceinline__ void fx_vol_adjoint(const McParams& p, long long* acc, unsigned* node, int nNodes,
                                               const FxInterval* sIv, const long long* sInv, int s, int lo, long long y,
                                               double av)
{
    const int nS = p.nS, nT = p.nT;
    const FxInterval iv = sIv[lo];
    const bool inner = lo > 0 && lo < nS;  // two knots; one at the flat ends
    // weight of the upper knot, units of 2^-59
    const long long t = inner ? fx_mul_add(sInv[lo], (long long)((unsigned long long)(y - iv.x) << iv.sh), 0) : 0;
    const int jl = lo - (lo > 0 ? 1 : 0);
    const longlong2 s0 = __ldg(reinterpret_cast<const longlong2*>(p.fx.step + s));
    const int2 col = __ldg(reinterpret_cast<const int2*>(&p.fx.step[s].colA));
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
        const int at = jl * nT;
        fx_node_add(node, nNodes, at + col.x, nL - lB, sft);
        fx_node_add(node, nNodes, at + col.y, lB, sft);
        if (inner)
        {
            fx_node_add(node, nNodes, at + nT + col.x, nR - rB, sft);
            fx_node_add(node, nNodes, at + nT + col.y, rB, sft);
        }
    }
    else
    {
        const double cR = c * ((double)t * 0x1p-59), cL = c - cR;
        const double tw = (double)s0.x * 0x1p-62;
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
__device__ __forceinline__ void fx_node_flush(long long* acc, unsigned* node, int nNodes, int threads)
{
    for (int i = threadIdx.x; i < nNodes; i += threads)
    {
        const unsigned n0 = node[i], n1 = node[i + nNodes], n2 = node[i + 2 * nNodes];
        if (n0 | n1 | n2)
        {
            node[i] = node[i + nNodes] = node[i + 2 * nNodes] = 0;
            const long long lo = (long long)(((unsigned long long)(n1 & 0xffu) << 32) | n0);  // 40 bits
            const long long hi = (long long)(((unsigned long long)n2 << 32) | n1) >> 8;
            if (hi) atomicAdd(reinterpret_cast<unsigned long long*>(&acc[2 * (1 + i)]), (unsigned long long)hi);
            if (lo) atomicAdd(reinterpret_cast<unsigned long long*>(&acc[2 * (1 + i) + 1]), (unsigned long long)lo);
        }
    }
}

}  // namespace cf
