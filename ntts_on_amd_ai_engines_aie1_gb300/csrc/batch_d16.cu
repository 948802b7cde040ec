// batch_d16.cu -- int16 instantiations of the direct batch kernel
// (batch_direct.cuh): one kernel per group of families; batch_k16.cu lists them
// in the configuration table.
#include "batch_direct.cuh"

namespace gbntt {

const void* batch_direct_i16(int el, int set, int occ, int cta) {
    constexpr int R2 = (1 << F_R2F16) | (1 << F_R2I16), R4 = 1 << F_R4F16, R8 = 1 << F_R8F16;
    constexpr int C16 = (1 << F_C16F) | (1 << F_C16I);
#define GB_K(CTA, EL, SET, OCC) \
    if (cta == CTA && el == EL && set == SET && occ == OCC) return reinterpret_cast<const void*>(&k_batch_direct<false, CTA, EL, SET, OCC>);
    GB_K(128, 4, R4, 10)
    GB_K(256, 4, R4, 6)
    GB_K(128, 4, R2, 10)
    GB_K(256, 4, R2, 5)
    GB_K(128, 4, R8, 10)
    GB_K(256, 4, R8, 5)
    GB_K(128, 4, C16, 10)
    GB_K(256, 4, C16, 6)
#undef GB_K
    return nullptr;
}

}  // namespace gbntt
