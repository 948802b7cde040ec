// kernels_tc16.cu -- per-plan launches of the tensor-core canonical int16
// transforms (tc16.cuh).
#include "tc16.cuh"

namespace gbntt {

namespace {

template <int LK, bool LB, bool SB>
__global__ void __launch_bounds__(TC_CTA, TC_OCC) k_tc16(const __grid_constant__ KArgs a, int L) {
    extern __shared__ __align__(128) unsigned char ring[];
    grid_dep_start();
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long w = (long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const long long tiles = ((a.batch << L) + TC_TILE - 1) / TC_TILE;
    if (w < tiles)
        tc_segment<LK, LB, SB>(a, L, w, tiles, warps, threadIdx.x & 31, ring + (threadIdx.x >> 5) * TC_WARP_RING);
}

template <int LK>
const void* for_mode(bool lb, bool sb) {
    return lb ? reinterpret_cast<const void*>(&k_tc16<LK, true, false>)
           : sb ? reinterpret_cast<const void*>(&k_tc16<LK, false, true>)
                : reinterpret_cast<const void*>(&k_tc16<LK, false, false>);
}

}  // namespace

const void* tc16_kernel(int L, bool bitrev_in, bool bitrev_out) {
    switch (tc_lk(L)) {
    case 8: return for_mode<8>(bitrev_in, bitrev_out);
    case 9: return for_mode<9>(bitrev_in, bitrev_out);
    default: return for_mode<10>(bitrev_in, bitrev_out);
    }
}

}  // namespace gbntt
