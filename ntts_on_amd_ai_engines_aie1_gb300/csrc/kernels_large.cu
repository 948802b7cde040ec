// kernels_large.cu -- int32 lane transforms of 2^14 .. 2^22 coefficients in two passes.
//
// The reference's layers are in-place butterflies on position bits (see
// device.cuh).  For n = 2^(L1 + L2), the forward layers on the L1 high bits
// touch, for each fixed low part c, only the positions (j << L2) | c; their
// twiddle block is j's bits above the butterfly, independent of c.  So the
// first L1 layers are 2^L2 independent L1-bit sub-transforms over "columns"
// (stride 2^L2), and the last L2 layers are 2^L1 sub-transforms over
// contiguous "rows" whose block index is (row << L2 | s) >> (bit + 1).  The
// inverse (Gentleman-Sande, low bits first) runs rows first, then columns.
// Every butterfly keeps the reference's arithmetic, so outputs stay bit-exact.
#include "device.cuh"

namespace gbntt {

namespace {

// 16 coefficients per thread (measured against 32 on GB300, same box: n = 2^20
// forward 0.77 vs 0.86 ms, inverse 0.67 vs 0.85 ms for 64 polynomials)
constexpr int LARGE_EL = 4;
__host__ __device__ constexpr int large_el(int L) { return L < LARGE_EL ? L : LARGE_EL; }
// At least 32 columns (128-byte accesses) and 256 threads per CTA.  Rows are
// 2^12 coefficients (2^13 for n = 2^22), as long as the row pass runs well;
// columns are the rest, so that their pass has two windows at most and at least
// four bits.  2^14, 2^17 and 2^18 measured faster with shorter rows (over 2^26 coefficients, forward /
// inverse: 2^17 5+12 391/406 us, 7+10 390/386; 2^18 6+12 410/421, 7+11 408/409;
// 64 polynomials of 2^14, 4+10 16/13 us, 5+9 14/13).
__host__ __device__ constexpr int large_cols(int L1) {
    const int c = 256 >> (L1 - large_el(L1));
    return c < 32 ? 32 : c;
}

// Rows per CTA: one, and for the inverse, whose first pass this is, as many as
// make 128 threads, with registers for six such CTAs per SM.  With 64 threads (2^17) and
// 32 (2^14) short calls took 4 us longer: 2 / 4 / 8 polynomials of 2^17 11.1 /
// 11.6 / 15.2 us for 16.9 / 17.0 / 19.1, 16 / 64 of 2^14 10.9 / 14.6 for 14.9 /
// 18.0; 512 of 2^17 369 for 369 (373 with registers for ten).  The forward's rows,
// its second pass, do not gain (8 of 2^17 17.3 for 15.9).
__host__ __device__ constexpr int large_rows(int fam, int L2) {
    const int G = 1 << (L2 - LARGE_EL);
    return topdown(fam) || G >= 128 ? 1 : 128 / G;
}
__host__ __device__ constexpr int large_row_blocks(int fam, int L2, int rows) {
    return rows > 1 ? 6 : kntt_min_blocks(fam, 1 << (L2 - LARGE_EL), LARGE_EL);
}

// one CTA: COLS adjacent columns of one polynomial, G threads per column
template <int FAM, int L1, int COLS>
__global__ void __launch_bounds__(COLS << (L1 - large_el(L1)), kntt_min_blocks(FAM, COLS << (L1 - large_el(L1)), LARGE_EL))
    k_cols(const __grid_constant__ KArgs a, int L2) {
    constexpr int EL = large_el(L1), G = 1 << (L1 - EL), E = 1 << EL, NS = nsteps(FAM, L1);
    constexpr int LO0 = window_lo(FAM, L1, EL, 0), LOZ = window_lo(FAM, L1, EL, NS - 1);
    extern __shared__ int csmem[];
    grid_dep_start();
    const int tid = threadIdx.x, cl = tid % COLS, g = tid / COLS;
    const long long blocks_per_poly = (1LL << L2) / COLS;
    const long long block = pass_block(topdown(FAM));
    const long long poly = block / blocks_per_poly;
    const long long c0 = (block % blocks_per_poly) * COLS;
    const long long base = (poly << (L1 + L2)) + c0 + cl;
    const int* in = static_cast<const int*>(a.in) + base;
    int* out = static_cast<int*>(a.out) + base;
    int v[E];
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = in[(long long)posmap<LO0, EL>(g, k) << L2];
    const KC kc = make_kc(a);
    run_steps_x<FAM, L1, EL, COLS, false>(v, csmem, g, kc, 0, cl, std::make_integer_sequence<int, NS>{});
    epilogue_all<false>(v, a);
    __syncthreads();   // every read of `in` is done before an in-place store lands
#pragma unroll
    for (int k = 0; k < E; ++k) out[(long long)posmap<LOZ, EL>(g, k) << L2] = v[k];
}

// one CTA: P rows of 2^L2 coefficients, G threads per row
template <int FAM, int L2, int P>
__global__ void __launch_bounds__(P << (L2 - LARGE_EL), large_row_blocks(FAM, L2, P))
    k_rows(const __grid_constant__ KArgs a, int L1) {
    constexpr int EL = LARGE_EL, G = 1 << (L2 - EL), E = 1 << EL, NS = nsteps(FAM, L2), N = 1 << L2;
    constexpr int LO0 = window_lo(FAM, L2, EL, 0), LOZ = window_lo(FAM, L2, EL, NS - 1);
    extern __shared__ int rsmem[];
    grid_dep_start();
    const int tid = threadIdx.x, lp = tid / G, g = tid % G;
    const long long row = (long long)pass_block(!topdown(FAM)) * P + lp;        // rows of all polynomials, in order
    const bool active = row < (a.batch << L1);
    const int hi = (int)(row & ((1LL << L1) - 1));               // row index inside its polynomial
    int* sp = rsmem + lp * xwords(L2);
    int v[E];
    if (active) {
        load_poly<true, L2, EL, LO0>(v, a, row, g);
    } else {
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] = 0;
    }
    const KC kc = make_kc(a);
    run_steps_x<FAM, L2, EL, 0, true>(v, sp, g, kc, hi, 0, std::make_integer_sequence<int, NS>{});
    epilogue_all<false>(v, a);
    if (active) store_poly<true, L2, EL, LOZ>(v, a, row, g);
}

template <int FAM, int L1, int L2>
LargeInfo make_large() {
    LargeInfo li;
    li.L1 = L1;
    li.L2 = L2;
    constexpr int EL1 = large_el(L1), C = large_cols(L1);
    li.cols = reinterpret_cast<const void*>(&k_cols<FAM, L1, C>);
    li.cols_threads = C << (L1 - EL1);
    li.cols_smem = num_windows(FAM, L1, EL1) > 1 ? C * (1 << L1) * 4 : 0;
    li.cols_per_cta = C;
    constexpr int G2 = 1 << (L2 - LARGE_EL), P = large_rows(FAM, L2);
    li.rows = reinterpret_cast<const void*>(&k_rows<FAM, L2, P>);
    li.rows_threads = P * G2;
    li.rows_smem = P * xwords(L2) * 4;
    li.rows_per_cta = P;
    return li;
}

template <int FAM>
LargeInfo large_for(int L) {
    switch (L) {
    case 14: return make_large<FAM, 5, 9>();
    case 15: return make_large<FAM, 4, 11>();
    case 16: return make_large<FAM, 4, 12>();
    case 17: return make_large<FAM, 7, 10>();
    case 18: return make_large<FAM, 7, 11>();
    case 19: return make_large<FAM, 7, 12>();
    case 20: return make_large<FAM, 8, 12>();
    case 21: return make_large<FAM, 9, 12>();
    case 22: return make_large<FAM, 9, 13>();
    default: return LargeInfo();
    }
}

}  // namespace

LargeInfo large_info(int fam, int L) {
    if (fam == F_R2F32) return large_for<F_R2F32>(L);
    if (fam == F_R2G32) return large_for<F_R2G32>(L);
    return LargeInfo();
}

}  // namespace gbntt
