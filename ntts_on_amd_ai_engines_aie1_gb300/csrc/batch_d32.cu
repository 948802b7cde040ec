// batch_d32.cu -- int32 instantiations of the direct batch kernel
// (batch_direct.cuh); batch_k32.cu lists them in the configuration table.
#include "batch_direct.cuh"

namespace gbntt {

const void* batch_direct_i32(int el, int set, int occ, int cta) {
    constexpr int K32 = (1 << F_R2F32) | (1 << F_R2G32), C32 = (1 << F_C32F) | (1 << F_C32I);
#define GB_K(CTA, EL, SET, OCC) \
    if (cta == CTA && el == EL && set == SET && occ == OCC) return reinterpret_cast<const void*>(&k_batch_direct<true, CTA, EL, SET, OCC>);
    GB_K(128, 4, K32, 10)
    GB_K(256, 4, K32, 5)
    GB_K(256, 5, K32, 4)
    GB_K(512, 4, K32, 2)
    GB_K(128, 4, C32, 10)
    GB_K(256, 4, C32, 5)
    GB_K(256, 5, C32, 4)
    GB_K(512, 4, C32, 2)
#undef GB_K
    return nullptr;
}

}  // namespace gbntt
