// Instantiations of the radix-2 int16 transform kernels (forward and inverse).
#include "device.cuh"

namespace gbntt {

#define GB_CASE(F, L) case L: return make_kernel_info<F, L, false>();
// the latency form of design F at L, or none
#define GB_LAT(F, L) case L: if constexpr (has_lat(F, L)) return make_kernel_info<F, L, false, true>(); else return KernelInfo();

// At n = 4 and 8 a kernel for each form of the butterflies: with the three in one
// kernel, choosing costs n = 8 a tenth (moduli above 2^14, us over 2^25
// coefficients: forward 35.5 for 40.4, inverse 32.4 for 36.4; q = 12289 32.3 for
// 34.4 and 30.9 for 32.2) and n = 4 3 % (39.1 for 40.4).
#define GB_FORMS(F, L)                                                                             \
    case L:                                                                                        \
        return form == R2_LEAN_ODD ? make_kernel_info<F, L, false, false, R2_LEAN_ODD>()           \
               : form == R2_LEAN   ? make_kernel_info<F, L, false, false, R2_LEAN>()               \
                                   : make_kernel_info<F, L, false, false, R2_WIDE>();

KernelInfo kinfo_r2f16(int L, bool lat, int form) {
    if (lat) {
        switch (L) {
            GB_LAT(F_R2F16, 9) GB_LAT(F_R2F16, 10) GB_LAT(F_R2F16, 11) GB_LAT(F_R2F16, 12)
            default: return KernelInfo();
        }
    }
    switch (L) {
        GB_CASE(F_R2F16, 1) GB_FORMS(F_R2F16, 2) GB_FORMS(F_R2F16, 3) GB_CASE(F_R2F16, 4)
        GB_CASE(F_R2F16, 5) GB_CASE(F_R2F16, 6) GB_CASE(F_R2F16, 7) GB_CASE(F_R2F16, 8)
        GB_CASE(F_R2F16, 9) GB_CASE(F_R2F16, 10) GB_CASE(F_R2F16, 11) GB_CASE(F_R2F16, 12)
        default: return KernelInfo();
    }
}

KernelInfo kinfo_r2i16(int L, bool lat, int form) {
    if (lat) {
        switch (L) {
            GB_LAT(F_R2I16, 9) GB_LAT(F_R2I16, 10) GB_LAT(F_R2I16, 11) GB_LAT(F_R2I16, 12)
            default: return KernelInfo();
        }
    }
    switch (L) {
        GB_CASE(F_R2I16, 1) GB_FORMS(F_R2I16, 2) GB_FORMS(F_R2I16, 3) GB_CASE(F_R2I16, 4)
        GB_CASE(F_R2I16, 5) GB_CASE(F_R2I16, 6) GB_CASE(F_R2I16, 7) GB_CASE(F_R2I16, 8)
        GB_CASE(F_R2I16, 9) GB_CASE(F_R2I16, 10) GB_CASE(F_R2I16, 11) GB_CASE(F_R2I16, 12)
        default: return KernelInfo();
    }
}

}  // namespace gbntt
