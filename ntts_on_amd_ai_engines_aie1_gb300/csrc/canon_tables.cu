// canon_tables.cu -- twiddle tables of the canonical families, computed on
// the device at plan creation and kept resident.
//
// Every entry is a pair (w, w') with w = root^e mod q in [0, q) and
// w' = floor(w 2^32 / q), the quotient Shoup's multiplication needs.  Each
// thread computes its entries independently (square-and-multiply with 64-bit
// products), so the tables need no host arithmetic and no upload.
#include "canon_tables.h"

namespace gbntt {

namespace {

__device__ __forceinline__ unsigned mulmod(unsigned a, unsigned b, unsigned q) {
    return (unsigned)(((unsigned long long)a * b) % q);
}

__device__ unsigned powmod_dev(unsigned b, unsigned long long e, unsigned q) {
    unsigned r = 1u % q;
    while (e) {
        if (e & 1) r = mulmod(r, b, q);
        b = mulmod(b, b, q);
        e >>= 1;
    }
    return r;
}

__device__ __forceinline__ int2 shoup_pair(unsigned w, unsigned q) {
    return make_int2((int)w, (int)(unsigned)(((unsigned long long)w << 32) / q));
}

// n entries: entry 2^B + j = root^(+-j 2^(L-1-B)) (+ forward, - inverse), the
// twiddle of the layer on bit B at low position bits j; entry 0 = 1.
__global__ void k_canon_table(int2* tab, int L, unsigned q, unsigned root, int inverse) {
    const int n = 1 << L;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        unsigned long long e = 0;
        if (i > 0) {
            const int B = 31 - __clz(i);
            const unsigned long long j = (unsigned long long)(i - (1 << B));
            e = (j << (L - 1 - B)) & (unsigned long long)(n - 1);
            if (inverse && e) e = (unsigned long long)n - e;
        }
        tab[i] = shoup_pair(powmod_dev(root, e, q), q);
    }
}

// the tail's words of the layer on bit 0, which hold every block's entry
// (canon_tables.h): the right one of two neighbours is the left one times
// root^(+-bitrev(1)) = root^(+-n/4)
__global__ void k_tail_all(int4* tail, int L, int L2, int EL, unsigned q, unsigned root, int inverse) {
    const int n = 1 << L, g2 = L2 - EL, w2 = EL - 2;          // log2 threads of a row, words of the layer
    const unsigned quarter = powmod_dev(root, inverse ? 3u * (unsigned)(n / 4) : (unsigned)(n / 4), q);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 4; i += gridDim.x * blockDim.x) {
        const int g = i & ((1 << g2) - 1), word = (1 << w2) - 1 + ((i >> g2) & ((1 << w2) - 1)), r = i >> (g2 + w2);
        unsigned long long e = __brev((unsigned)two_pass_tail_block(L2, EL, r, word, g)) >> (33 - L);
        if (inverse && e) e = (unsigned long long)n - e;
        const unsigned w = powmod_dev(root, e, q);
        const int2 x = shoup_pair(w, q), y = shoup_pair(mulmod(w, quarter, q), q);
        tail[two_pass_tail_at(L2, EL, r, word, g)] = make_int4(x.x, x.y, y.x, y.y);
    }
}

// the block table and the tail's other words, copied from those
__global__ void k_two_pass_rest(int2* blocks, int4* tail, int L, int L2, int EL) {
    const int g2 = L2 - EL, rest = (1 << (EL - 2)) - 1;       // words of the other layers
    const long long nb = (long long)two_pass_blocks(L) / 2, count = nb + ((long long)rest << (L - EL));
    for (long long i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        if (i < nb) {
            reinterpret_cast<int4*>(blocks)[i] = tail[two_pass_tail_of(L2, EL, (int)(2 * i))];
        } else {
            const int j = (int)(i - nb), g = j & ((1 << g2) - 1), word = (j >> g2) % rest, r = (j >> g2) / rest;
            tail[two_pass_tail_at(L2, EL, r, word, g)] =
                tail[two_pass_tail_of(L2, EL, two_pass_tail_block(L2, EL, r, word, g))];
        }
    }
}

int grid_of(long long count) {
    long long b = (count + 255) / 256;
    return (int)(b < 1 ? 1 : (b > 4096 ? 4096 : b));
}

}  // namespace

size_t canon_table_entries(int L, bool) { return (size_t)1 << L; }

cudaError_t make_canon_table(int2* d_tab, int L, uint32_t q, uint32_t root, bool inverse, cudaStream_t s) {
    k_canon_table<<<grid_of((long long)canon_table_entries(L, inverse)), 256, 0, s>>>(d_tab, L, q, root,
                                                                                    inverse ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t make_two_pass_tables(int2* d_tab, int L, int L2, int EL, uint32_t q, uint32_t root, bool inverse,
                                 cudaStream_t s) {
    int4* tail = reinterpret_cast<int4*>(d_tab + two_pass_blocks(L));
    const int grid = grid_of(1ll << (L - 2));
    k_tail_all<<<grid, 256, 0, s>>>(tail, L, L2, EL, q, root, inverse ? 1 : 0);
    k_two_pass_rest<<<grid, 256, 0, s>>>(d_tab, tail, L, L2, EL);
    return cudaGetLastError();
}

}  // namespace gbntt
