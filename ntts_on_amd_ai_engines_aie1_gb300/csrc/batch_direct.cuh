// batch_direct.cuh -- the batch kernel without staging: one CTA per share of a
// tile, each polynomial from global memory to registers and back as in the
// per-plan kernels (instantiated in batch_d16.cu and batch_d32.cu, launched by
// batch.cu).
//
// The persistent kernel (batch_kernel.cuh) moves every tile through a shared
// stage with bulk copies and pays for it with 2 x 16 KB per CTA and two more
// passes over shared memory; since the per-plan kernels run at 40 warps per SM
// the warps hide the loads by themselves.  A CTA finds its segment with one
// warp-wide search and reads the arguments where they are.
//
// The unit of the tile order stays the persistent kernel's (256 threads' worth
// of polynomials); a 128-thread CTA takes half of it, a 512-thread one has its
// own.
#pragma once

#include "batch_kernel.cuh"

namespace gbntt {

template <bool I32, int CTA, int ELMAX, int SET, int OCC>
__global__ void __launch_bounds__(CTA, OCC) k_batch_direct(const BatchDev b, int) {
    grid_dep_start();
    extern __shared__ int dsmem[];
    constexpr int SPLIT = direct_unit(CTA) / CTA;
    const long long t = blockIdx.x / SPLIT;
    const SegDev* sd = &b.segs[warp_seg_find(b, t, 0, threadIdx.x & 31)];
    const KArgs& a = sd->a;
    const long long poly0 = ((t - sd->tile0) * SPLIT + blockIdx.x % SPLIT) * (long long)(sd->polys_per_tile / SPLIT);
    if (poly0 >= a.batch) return;
    switch (sd->variant) {
#define GB_CASE(F, L)                                                                                        \
    case variant_id(F, L):                                                                                   \
        if constexpr (fam_i32(F) == I32 && ((SET >> F) & 1) && batch_fits(L, CTA, ELMAX))                    \
            ntt_tile<F, L, batch_el(L, ELMAX), (CTA >> (L - batch_el(L, ELMAX))), false>(a, a.lean, poly0, dsmem); \
        break;
        GB_ALL_VARIANTS(GB_CASE)
#undef GB_CASE
        default: break;
    }
}

}  // namespace gbntt
