// Instantiations of dupire_fx64 for one product (two units, compiled in parallel).
#include "mc_dupire_fx64.cuh"

namespace cf {

const void* dupire_fx64_ptr_european(int rng, int risk, int block)
{
#define CF_K(RG, RK, RB) \
    if (rng == RG && risk == RK && block == RB) return (const void*)&dupire_fx64<PROD_EUROPEAN, RG, RK, RB>;
    CF_K(RNG_MRG, false, 128)
    CF_K(RNG_MRG, true, 128)
    CF_K(RNG_MRG, true, 384)
    CF_K(RNG_SOBOL, false, 128)
    CF_K(RNG_SOBOL, true, 128)
    CF_K(RNG_SOBOL, true, 384)
#undef CF_K
    return nullptr;
}

}  // namespace cf
