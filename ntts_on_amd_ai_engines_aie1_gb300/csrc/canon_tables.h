// canon_tables.h -- device-built twiddle tables of the canonical families
// (canon_tables.cu).
#pragma once

#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>

namespace gbntt {

// (w, floor(w 2^32 / q)) pairs, n entries: root^(+-j 2^(L-1-B)) at 2^B + j
size_t canon_table_entries(int L, bool inverse);
cudaError_t make_canon_table(int2* d_tab, int L, uint32_t q, uint32_t root, bool inverse, cudaStream_t s);

// The tables of a two-pass transform (kernels_c32_large.cu) of 2^L coefficients,
// rows of 2^L2, 2^EL coefficients per thread in the row pass.  A butterfly's
// block b, the position bits above its own, has the entry root^(+-bitrev(b)),
// log2(n) - 1 bits reversed; n / 2 blocks in all.
//   blocks: the entries of the first n / 8, by block.  They serve the column
//     pass and the layers on bit 2 and above of the rows;
//   tail: a row's layers on its lowest bits, all EL - 1 of them that have two
//     or more blocks in a thread's run, in the order in which its threads read
//     them: 16-byte words of two neighbouring blocks, [row][word][thread],
//     2^(EL-1) - 1 words a thread, those of the layer on bit B from 2^(EL-2-B) - 1.
// 8 bytes a coefficient together (n / 8 entries, 7 n / 16 words).
__host__ __device__ constexpr size_t two_pass_blocks(int L) { return (size_t)1 << (L - 3); }
__host__ __device__ constexpr int two_pass_tail_words(int EL) { return (1 << (EL - 1)) - 1; }
// entries of both: n / 8 and two for each word
__host__ __device__ constexpr size_t two_pass_entries(int L, int EL) {
    return two_pass_blocks(L) + 2 * ((size_t)two_pass_tail_words(EL) << (L - EL));
}
// the word of thread g of row r
__host__ __device__ constexpr long long two_pass_tail_at(int L2, int EL, int r, int word, int g) {
    return (((long long)r * two_pass_tail_words(EL) + word) << (L2 - EL)) + g;
}
// the first of its two blocks: words 2^p - 1 .. 2^(p+1) - 2 are the layer on bit EL - 2 - p
__host__ __device__ constexpr int two_pass_tail_block(int L2, int EL, int r, int word, int g) {
    int p = 0;
    while ((2 << p) <= word + 1) ++p;
    return (((r << (L2 - EL)) | g) << (p + 1)) | 2 * (word + 1 - (1 << p));
}
// where block b lies among the words of the layer on bit 0, which holds all of them
__host__ __device__ constexpr long long two_pass_tail_of(int L2, int EL, int b) {
    const int row_blocks = L2 - 1, run = EL - 1;      // log2: of a row's and of a thread's blocks
    return two_pass_tail_at(L2, EL, b >> row_blocks, (1 << (EL - 2)) - 1 + ((b & ((1 << run) - 1)) >> 1),
                            (b & ((1 << row_blocks) - 1)) >> run);
}
cudaError_t make_two_pass_tables(int2* d_tab, int L, int L2, int EL, uint32_t q, uint32_t root, bool inverse,
                                 cudaStream_t s);

}  // namespace gbntt
