// batch_tc16.cu -- the persistent batch kernel of the tensor-core canonical
// int16 transforms (tc16.cuh); batch_k16.cu lists it in the configuration table.
#include "batch_kernel.cuh"
#include "tc16.cuh"

namespace gbntt {

namespace {

// Every warp takes the tiles (1024 coefficients of one segment) at its own
// index modulo the launch's warps, in order; the tiles are equal work, so no
// counter hands them out.  Consecutive warp indices lie on different CTAs, so
// a batch of few tiles spreads over the SMs.
__global__ void __launch_bounds__(TC_CTA, TC_OCC) k_batch_tc16(const BatchDev b, int) {
    __shared__ __align__(128) unsigned char rings[TC_CTA / 32][TC_WARP_RING];
    unsigned char* ring = rings[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    grid_dep_start();
    const long long warps = (long long)gridDim.x * (TC_CTA / 32);
    long long t = (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    int s = 0;
    while (t < b.total_tiles) {
        s = warp_seg_find(b, t, s, lane);
        const SegDev* sd = &b.segs[s];
        const long long first = t - sd->tile0, tiles = sd->tiles;
        const KArgs& a = sd->a;
        const int L = sd->variant & 15, fam = sd->variant >> 4;
        // mode: 0 natural in, bit-reversed out; 1 natural in and out; 2 bit-reversed in, natural out
        const int mode = fam == F_C16F ? (a.natural_out ? 1 : 0) : (a.natural_in ? 1 : 2);
        switch (tc_lk(L) * 4 + mode) {
#define GB_TC(LK)                                                                                  \
    case LK * 4 + 0: tc_segment<LK, false, true>(a, L, first, tiles, warps, lane, ring); break;          \
    case LK * 4 + 1: tc_segment<LK, false, false>(a, L, first, tiles, warps, lane, ring); break;         \
    case LK * 4 + 2: tc_segment<LK, true, false>(a, L, first, tiles, warps, lane, ring); break;
            GB_TC(8)
            GB_TC(9)
            GB_TC(10)
#undef GB_TC
            default: break;
        }
        t += (tiles - first + warps - 1) / warps * warps;
    }
}

}  // namespace

const void* batch_kernel_tc16() { return reinterpret_cast<const void*>(&k_batch_tc16); }

}  // namespace gbntt
