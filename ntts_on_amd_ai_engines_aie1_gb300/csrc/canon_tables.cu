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

// 2^(L-1) entries: entry b = root^(+-bitrev(b)), L - 1 bits reversed
__global__ void k_block_table(int2* tab, int L, unsigned q, unsigned root, int inverse) {
    const int n = 1 << L;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += gridDim.x * blockDim.x) {
        unsigned long long e = __brev((unsigned)i) >> (33 - L);
        if (inverse && e) e = (unsigned long long)n - e;
        tab[i] = shoup_pair(powmod_dev(root, e, q), q);
    }
}

// the tail (see canon_tables.h), from the block table
__global__ void k_tail_table(int4* tail, const int2* tab, int L, int L2, int EL) {
    const int g2 = L2 - EL;                                   // log2 threads of a row
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 1 << (L - 1); i += gridDim.x * blockDim.x) {
        const int g = i & ((1 << g2) - 1), pair = (i >> g2) & ((1 << (EL - 1)) - 1), r = i >> (L2 - 1);
        const int p = 31 - __clz(pair + 1), B = EL - 2 - p;   // 2^p pairs on bit B
        if (B < 0) continue;                                  // the last word of each thread is unused
        const int2* t = tab + ((((r << g2) | g) << (p + 1)) | 2 * (pair + 1 - (1 << p)));
        tail[i] = make_int4(t[0].x, t[0].y, t[1].x, t[1].y);
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

size_t two_pass_entries(int L) { return ((size_t)1 << (L - 1)) + ((size_t)1 << L); }

cudaError_t make_two_pass_tables(int2* d_tab, int L, int L2, int EL, uint32_t q, uint32_t root, bool inverse,
                                 cudaStream_t s) {
    const int grid = grid_of(1ll << (L - 1));
    k_block_table<<<grid, 256, 0, s>>>(d_tab, L, q, root, inverse ? 1 : 0);
    k_tail_table<<<grid, 256, 0, s>>>(reinterpret_cast<int4*>(d_tab + ((size_t)1 << (L - 1))), d_tab, L, L2, EL);
    return cudaGetLastError();
}

}  // namespace gbntt
