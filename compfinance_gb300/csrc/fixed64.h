// 64-bit integer arithmetic of the fixed-point sums, for device code and its host tests.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define CF_HD __host__ __device__ __forceinline__
#else
#define CF_HD inline
#endif

namespace cf {

// The double with bits b as hi 2^-20 + lo 2^-60, rounded to units of 2^-60 (ties to even); false
// when |v| >= 2^42 (infinities and NaN included), which the caller converts in floating point.
CF_HD bool fix_split_bits(unsigned long long b, long long& hi, long long& lo)
{
    const int E = int(unsigned(b >> 32) >> 20) & 0x7ff;
    if (E >= 1023 + 42) return false;
    const unsigned long long m = (b & 0xfffffffffffffULL) | (E ? 0x10000000000000ULL : 0ULL);
    const int sh = E - 1015;  // |v| 2^60 = m 2^sh
    long long h = 0, l = 0;
    if (sh >= 40)
        h = (long long)(m << (sh - 40));
    else if (sh >= 0)
    {
        const int r = 40 - sh;
        h = (long long)(m >> r);
        l = (long long)((m & ((1ULL << r) - 1)) << sh);
    }
    else if (sh >= -54)
    {
        const unsigned long long half = 1ULL << (-sh - 1), rem = m & (2 * half - 1);
        l = (long long)(m >> -sh);
        l += (rem > half || (rem == half && (l & 1))) ? 1 : 0;
    }
    const bool neg = (long long)b < 0;
    hi = neg ? -h : h;
    lo = neg ? -l : l;
    return true;
}

}  // namespace cf
