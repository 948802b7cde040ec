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

// the tables of a two-pass transform (kernels_c32_large.cu): n / 2 entries
// root^(+-bitrev(b)) at b, its log2(n) - 1 bits reversed, then the tail, n / 2
// 16-byte words: for row r the entries of its layers on the lowest EL bits in
// pairs, [r][pair][thread] with 2^(EL-1) pairs for each of the 2^(L2-EL) threads
// (pair 2^(EL-2-B) - 1 + i: the blocks 2 i and 2 i + 1 of the thread on bit B)
size_t two_pass_entries(int L);
cudaError_t make_two_pass_tables(int2* d_tab, int L, int L2, int EL, uint32_t q, uint32_t root, bool inverse,
                                 cudaStream_t s);

}  // namespace gbntt
