// kernels_c32_large.cu -- canonical int32 transforms of 2^14 .. 2^22
// coefficients in two passes (columns, rows).
//
// Forward: Cooley-Tukey layers on natural-order input, high position bits
// first.  The block of a butterfly on bit B (the position bits above B) has the
// twiddle root^bitrev(block), the bits reversed as log2(n) - 1 of them, whatever
// the layer: the layer splits x^m - z^2 into x^(m/2) -+ z, and the root of a
// block's left half is the next layer's entry at twice its index.  With n = n1
// n2 and the polynomial viewed as n1 rows of n2 coefficients (row-major, no
// transpose in memory), the layers on the high bits are transforms of the
// columns, the same for every column, and those on the low bits are transforms
// of the rows, whose block index carries the row in its top bits.  One set of n / 2
// pairs serves all of them, and nothing is multiplied between the passes.  A
// row's entries for its lowest bits lie in the order in which its threads read
// them (the tail: 16 coalesced bytes a lane); the block table needs the first n
// / 8 pairs beside it, 8 bytes a coefficient together (canon_tables.h).
// The inverse (bit-reversed in, natural out, no n^-1) undoes the layers from the
// low bits up (Gentleman-Sande, root^-bitrev(block)): rows, then columns.
// Polynomials go through both passes in chunks of at most large_chunk_bytes().
//
// The column pass moves 2D tiles (COLS adjacent columns x n1 rows) between
// global and shared memory with the Tensor Memory Accelerator
// (cp.async.bulk.tensor.2d, an mbarrier with a bounded wait for the load, a
// bulk-group store); with lane = column every shared-memory access of a warp
// touches 32 distinct banks.  The row pass reads and writes whole rows with
// coalesced accesses.
//
// What bounds it: a butterfly's one high and two low 32-bit products hold the
// multiply pipe for 7.6 clocks a warp, 56 % of a 2^12 row pass; its loads and
// exchanges share the other half with the additions.  Over 2^26 coefficients,
// forward / inverse, against the four-step that multiplies by a twist between
// the passes (one factor per coefficient up to 2^20, two beyond), in chunks of 96
// MiB:
//   2^16 224/229 -> 224/214 us    2^18 237/239 -> 230/224
//   2^20 275/264 -> 265/256       2^22 317/322 -> 314/313
// Without the tail (64 contiguous bytes a lane): 2^16 236/225, 2^20 269/264.  All
// at once (large_chunk_bytes, pass_block): 2^16 200/190, 2^18 205/196, 2^20
// 237/225, 2^22 280/274.
#include <cuda.h>

#include "canon_tables.h"
#include "device.cuh"
#include "persist.cuh"

namespace gbntt {

namespace {

constexpr int ROW_EL = 4;            // 16 coefficients per thread in the row pass

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c, int r,
                                            unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_addr(dst)),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(c), "r"(r), "r"(smem_addr(bar))
        : "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int c, int r, const void* src) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<unsigned long long>(map)),
                 "r"(c), "r"(r), "r"(smem_addr(src))
                 : "memory");
}

// the column pass: COLS adjacent columns x N1 rows of one polynomial per CTA,
// G = N1 / 2^EL threads per column
template <int FAM, int L1, int EL, int COLS>
__global__ void __launch_bounds__(COLS << (L1 - EL))
    k_ccols(const __grid_constant__ CUtensorMap min, const __grid_constant__ CUtensorMap mout,
            const __grid_constant__ KArgs a, int n2, long long tile0, unsigned* err) {
    constexpr int E = 1 << EL, N1 = 1 << L1, NS = nsteps(FAM, L1);
    constexpr int R = N1 < 256 ? N1 : 256, NB = N1 / R;       // TMA boxes of at most 256 rows
    constexpr int LO0 = window_lo(FAM, L1, EL, 0), LOZ = window_lo(FAM, L1, EL, NS - 1);
    constexpr bool FWD = topdown(FAM);
    extern __shared__ __align__(128) unsigned char csm[];
    int* tile = reinterpret_cast<int*>(csm);
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(csm + N1 * COLS * 4);
    const int tid = threadIdx.x, cl = tid % COLS, g = tid / COLS;
    const long long tpp = n2 / COLS;                           // column tiles per polynomial
    const long long t = tile0 + pass_block(FWD);
    const int c0 = (int)((t % tpp) * COLS);
    const int r0 = (int)((t / tpp) * N1);
    if (tid == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    grid_dep_start();
    if (tid == 0) {
        mbar_expect_tx(bar, N1 * COLS * 4);
#pragma unroll
        for (int b = 0; b < NB; ++b) tma_load_2d(tile + b * R * COLS, &min, c0, r0 + b * R, bar);
    }
    const bool ok = mbar_wait(bar, 0);
    if (!__syncthreads_and(ok)) {
        // the tile did not arrive in time: record it, let the copy land, stop
        if (tid == 0) {
            atomicOr(err, 1u);
            mbar_wait(bar, 0);
        }
        return;
    }
    int v[E];
#pragma unroll
    for (int k = 0; k < E; ++k) v[k] = tile[posmap<LO0, EL>(g, k) * COLS + cl];
    if constexpr (FWD) prologue<FAM>(v, a);                    // raw input (the first pass)
    const KC kc = make_kc(a);
    run_steps_x<FAM, L1, EL, COLS, true>(v, tile, g, kc, 0, cl, std::make_integer_sequence<int, NS>{});
    if constexpr (!FWD) epilogue<FAM, false>(v, a);            // the inverse's last pass
    __syncthreads();                                           // every read of the tile is done
#pragma unroll
    for (int k = 0; k < E; ++k) tile[posmap<LOZ, EL>(g, k) * COLS + cl] = v[k];
    fence_proxy_async();                                       // visible to the bulk store
    __syncthreads();
    if (tid == 0) {
#pragma unroll
        for (int b = 0; b < NB; ++b) tma_store_2d(&mout, c0, r0 + b * R, tile + b * R * COLS);
        bulk_commit();
        bulk_wait_read();                                      // the tile is read before the CTA leaves
    }
}

// the row pass: one row of N2 coefficients per CTA of N2 / 2^EL threads; rows
// are numbered over the whole call, row r of its polynomial = r mod n1.
// The bound on resident threads caps the registers: 1536 (42 registers), 1024
// for rows of 2^10, where more of the loads fly at once (0.125 ms for the pass
// over 2^26 coefficients against 0.127 forward and 0.132 inverse with 1536).
constexpr int rows_min_blocks(int L2, int el) {
    const int b = (L2 <= 10 ? 1024 : 1536) >> (L2 - el);
    return b > 16 ? 16 : b;
}
// every layer that reads the block table is on bit 2 or above: its blocks are
// among the first n / 8
constexpr bool rows_blocks_held(int fam, int L2, int el) {
    for (int s = 0; s < nsteps(fam, L2); ++s) {
        const int b = step_b(fam, L2, s), lo = window_lo(fam, L2, el, s);
        if (b < 2 && (lo != 0 || b > el - 2)) return false;
    }
    return true;
}
template <int FAM, int L2, int EL>
__global__ void __launch_bounds__(1 << (L2 - EL), rows_min_blocks(L2, EL))
    k_crows(const __grid_constant__ KArgs a, int L1, long long row0) {
    constexpr int E = 1 << EL, N2 = 1 << L2, NS = nsteps(FAM, L2);
    constexpr int LO0 = window_lo(FAM, L2, EL, 0), LOZ = window_lo(FAM, L2, EL, NS - 1);
    constexpr bool FWD = topdown(FAM);
    static_assert((FWD ? LOZ : LO0) == 0, "contiguous runs at the rows' outer side");
    static_assert(rows_blocks_held(FAM, L2, EL), "the block table is too short for this split");
    extern __shared__ int rsm[];
    grid_dep_start();
    const int g = threadIdx.x;
    const long long row = row0 + pass_block(!FWD);
    const int r = (int)(row & ((1 << L1) - 1));
    int v[E];
    if constexpr (FWD) {
        // strided window: thread g holds columns g + G k
        const int* src = static_cast<const int*>(a.in) + row * N2;
#pragma unroll
        for (int k = 0; k < E; ++k) v[k] = src[posmap<LO0, EL>(g, k)];
    } else {
        load_poly<true, L2, EL, 0>(v, a, row, g);              // thread g: columns g E .. g E + E - 1
        prologue<FAM>(v, a);                                   // raw input (the first pass)
    }
    KC kc = make_kc(a);
    kc.tail = reinterpret_cast<const int4*>(a.tab + two_pass_blocks(L1 + L2)) + two_pass_tail_at(L2, EL, r, 0, g);
    run_steps_x<FAM, L2, EL, 0, true>(v, rsm, g, kc, r, 0, std::make_integer_sequence<int, NS>{}, true);   // rsm untouched so far
    if constexpr (FWD) {
        epilogue<FAM, false>(v, a);                            // the forward's last pass
        store_poly<true, L2, EL, 0>(v, a, row, g);
    } else {
        int* dst = static_cast<int*>(a.out) + row * N2;
#pragma unroll
        for (int k = 0; k < E; ++k) dst[posmap<LOZ, EL>(g, k)] = v[k];
    }
}

// The split of 2^L.  Short rows spread their exchange barriers over more CTAs
// of an SM (16 of 64 threads at 2^10, 6 of 256 at 2^12) as long as the columns
// stay within two windows (2^8).  Row passes alone over 2^26 coefficients,
// with a twist: 2^9 0.139 ms, 2^10 0.125, 2^11 0.137, 2^12 0.160, 2^13 0.211.
constexpr int split_l2(int L) { return L <= 18 ? 10 : (L == 19 ? 11 : 12); }
constexpr int col_el(int L1) { return L1 <= 7 ? (L1 < 4 ? L1 : 4) : 5; }
// Columns per CTA: two warps, at least 16 columns (64 bytes of a row), tiles of
// at most 32 KB.  Over 2^26 coefficients: 2^8 x 32 0.115 ms (16 coefficients per
// thread), x 16 0.102, x 8 0.116; 2^7 x 32 0.103, x 16 0.094; 2^5 x 32 0.091,
// x 16 0.139; 2^9 x 32 0.149, x 16 0.123; 2^10 x 16 0.160, x 8 0.148.
constexpr int col_width(int L1) {
    const int G = 1 << (L1 - col_el(L1)), w = 64 / G < 16 ? 16 : 64 / G;
    return (w << L1) > 8192 ? 8192 >> L1 : w;
}
template <int FAM, int L>
CanonLarge make_canon_large() {
    constexpr int L2 = split_l2(L), L1 = L - L2;
    constexpr int ELC = col_el(L1), COLS = col_width(L1);
    CanonLarge li;
    li.L1 = L1;
    li.row_el = ROW_EL;
    li.L2 = L2;
    li.cols = reinterpret_cast<const void*>(&k_ccols<FAM, L1, ELC, COLS>);
    li.cols_threads = COLS << (L1 - ELC);
    li.cols_smem = (1 << L1) * COLS * 4 + 16;
    li.cols_width = COLS;
    li.rows = reinterpret_cast<const void*>(&k_crows<FAM, L2, ROW_EL>);
    li.rows_threads = 1 << (L2 - ROW_EL);
    li.rows_smem = xwords(L2) * 4;
    return li;
}

template <int FAM>
CanonLarge canon_large_for(int L) {
    switch (L) {
    case 14: return make_canon_large<FAM, 14>();
    case 15: return make_canon_large<FAM, 15>();
    case 16: return make_canon_large<FAM, 16>();
    case 17: return make_canon_large<FAM, 17>();
    case 18: return make_canon_large<FAM, 18>();
    case 19: return make_canon_large<FAM, 19>();
    case 20: return make_canon_large<FAM, 20>();
    case 21: return make_canon_large<FAM, 21>();
    case 22: return make_canon_large<FAM, 22>();
    default: return CanonLarge();
    }
}

// cuTensorMapEncodeTiled (driver API, version 12000), reached through the runtime
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &qr) !=
                cudaSuccess ||
            qr != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// a 2D view of `rows` rows of n2 int32 coefficients, COLS x R boxes
cudaError_t make_map(CUtensorMap* map, const void* base, long long rows, int n2, int cols, int box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)n2, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)n2 * 4};
    const cuuint32_t box[2] = {(cuuint32_t)cols, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace

CanonLarge canon_large_info(int fam, int L) {
    if (fam == F_C32F) return canon_large_for<F_C32F>(L);
    if (fam == F_C32I) return canon_large_for<F_C32I>(L);
    return CanonLarge();
}

cudaError_t launch_canon_large(const CanonLarge& li, const KArgs& base, const int2* tab, const void* in, void* out,
                               long long batch, bool inverse, unsigned* err, cudaStream_t s, int* launches) {
    const int n1 = 1 << li.L1, n2 = 1 << li.L2;
    const long long n = (long long)n1 * n2;
    const int box_rows = n1 < 256 ? n1 : 256;
    CUtensorMap map_in, map_out;
    cudaError_t e = make_map(&map_out, out, batch * n1, n2, li.cols_width, box_rows);
    if (e != cudaSuccess) return e;
    // the forward's column pass reads the input; the inverse's runs in place
    if (!inverse && in != out) {
        e = make_map(&map_in, in, batch * n1, n2, li.cols_width, box_rows);
        if (e != cudaSuccess) return e;
    } else {
        map_in = map_out;
    }
    long long chunk = large_chunk_bytes() / (n * 4);
    if (chunk < 1) chunk = 1;
    const long long tpp = n2 / li.cols_width;
    KArgs ac = base, ar = base;
    ac.tab = tab;
    ar.tab = tab;
    int nl = 0;
    for (long long p0 = 0; p0 < batch; p0 += chunk) {
        const long long np = chunk < batch - p0 ? chunk : batch - p0;
        const long long tile0 = p0 * tpp, row0 = p0 * n1, rows = np * n1;
        int L1 = li.L1;
        // programmatic dependent launches (grid_dep_start); 2^22 runs 2 % faster
        // with the driver's own split of each pass
        const int share = li.L1 + li.L2 < 22 ? SMEM_SHARE : 0;
        auto launch = [&](const void* fn, unsigned grid, int threads, int smem, void** args) {
            ++nl;
            return launch_kernel(fn, grid, threads, smem, args, s, true, share);
        };
        auto cols = [&]() {
            void* args[] = {&map_in, &map_out, &ac, const_cast<int*>(&n2), const_cast<long long*>(&tile0), &err};
            return launch(li.cols, (unsigned)(np * tpp), li.cols_threads, li.cols_smem, args);
        };
        auto rowsk = [&](const void* src) {
            ar.in = src;
            ar.out = out;
            void* args[] = {&ar, &L1, const_cast<long long*>(&row0)};
            return launch(li.rows, (unsigned)rows, li.rows_threads, li.rows_smem, args);
        };
        if (!inverse) {
            e = cols();
            if (e == cudaSuccess) e = rowsk(out);
        } else {
            e = rowsk(in);
            if (e == cudaSuccess) e = cols();
        }
        if (e != cudaSuccess) return e;
    }
    if (launches) *launches = nl;
    return cudaSuccess;
}

}  // namespace gbntt
