// tc_tables.cpp -- host-built tables of the tensor-core transforms (tc16.cuh):
// the two DFT matrices as fp16 byte-limb fragments and the twiddle pairs, each
// in the order a warp's lanes read them.
#include "tc_tables.h"

#include "tables.h"

namespace gbntt {

namespace {

// fp16 bits of an integer of at most 11 significant bits
uint32_t f16_bits(int v) {
    if (!v) return 0;
    const uint32_t sign = v < 0 ? 0x8000u : 0u;
    uint32_t m = (uint32_t)(v < 0 ? -v : v);
    const int e = 31 - __builtin_clz(m);
    return sign | (uint32_t)(e + 15) << 10 | ((e <= 10 ? m << (10 - e) : m >> (e - 10)) & 0x3FFu);
}

// the centred residue's limbs 256 h + l as fp16 bits: hs h and 2 l
struct Limbs {
    uint32_t h, l;
};
Limbs limbs(uint32_t w, uint32_t q, int hs) {
    const int v = w > q / 2 ? (int)w - (int)q : (int)w;
    int l = v & 255;
    if (l >= 128) l -= 256;
    return {f16_bits(hs * ((v - l) / 256)), f16_bits(2 * l)};
}

struct Maps {
    int LK, l2, R1, R2;
    bool lb, sb;
    // input row (natural index u) of k-slot x of set s
    int u(int s, int x) const {
        if (!lb) return R1 == 32 ? 2 * x + s : x;
        const int t = (x & 7) >> 1, y = 4 * t + 2 * (x >> 3) + (x & 1);     // 4 t + {0, 1, 2, 3}
        return (int)bitrev((uint32_t)(16 * s + y), R1 == 32 ? 5 : 4);
    }
    // output row m (below 16) of tile row i
    int m(int i) const { return sb ? (int)bitrev((uint32_t)i, 4) : (i < 8 ? 2 * i : 2 * (i - 8) + 1); }
    // input column of n-tile j, slot v: polynomial of the unit and natural c
    void col(int j, int v, int* poly, int* c) const {
        if (LK > 8) {
            *poly = 0;
            *c = lb ? (int)bitrev((uint32_t)(8 * j + v), 5) : 4 * v + 2 * (j & 1) + (j >> 1);
            return;
        }
        const int x = lb ? 8 * j + v : 2 * v + j;
        *poly = x / R2;
        *c = lb ? (l2 ? (int)bitrev((uint32_t)(x % R2), l2) : 0) : x % R2;
    }
    // output column of tile jj, slot x: polynomial and natural v (below 16 for LK > 8)
    void out(int jj, int x, int* poly, int* v) const {
        const int t = x >> 1, e = x & 1;
        if (LK > 8) {
            *poly = 0;
            *v = sb ? (int)bitrev((uint32_t)(8 * t + 4 * jj + 2 * e), 5) : 8 * jj + x;
            return;
        }
        const int y = sb ? 4 * t + 2 * jj + e : 8 * jj + x;
        *poly = y / R2;
        *v = sb ? (l2 ? (int)bitrev((uint32_t)(y % R2), l2) : 0) : y % R2;
    }
};

}  // namespace

// The quotient of stage 2 (tc_reduce) is rounded twice: 1.5 2^23 - 1.5 2^23 / q
// is held as an integer, off by the distance d of 1.5 2^23 / q from one, and the
// product is rounded to an integer, with an argument off by less than 32 / q
// (the rounded sum and reciprocal).  The remainder stays inside (-q, q) when
// d + 1/2 + 32 / q is below one.
bool tc_supported(int L, int64_t q) {
    if (L < TC_MIN_L || L > TC_MAX_L || q >= 32768) return false;
    const int64_t r = 12582912 % q, d = r < q - r ? r : q - r;    // d / q from an integer
    return 2 * (d + 32) < q;
}

void tc_build(int L, int64_t modulus, int64_t root, bool inverse, bool natural, bool scale, std::vector<uint32_t>& out,
              uint32_t* ke, uint32_t* corr) {
    Maps M;
    M.LK = tc_lk(L);
    M.R1 = tc_r1(M.LK);
    M.R2 = (1 << L) / M.R1;
    M.l2 = L - (M.R1 == 32 ? 5 : 4);
    M.lb = inverse && !natural;
    M.sb = !inverse && !natural;
    const int S1 = tc_s1(M.LK), S2 = tc_s2(M.LK), NT = tc_cols(M.LK) / 8;
    // q < 2^15: every product below fits 32 bits
    const uint32_t n = 1u << L, q = (uint32_t)modulus;
    const uint32_t w0 = (uint32_t)(inverse ? modinv(root, modulus) : root);
    std::vector<uint32_t> pw(n);                      // powers of the root
    pw[0] = 1 % q;
    for (uint32_t i = 1; i < n; ++i) pw[i] = pw[i - 1] * w0 % q;
    auto power = [&](int e) { return pw[(uint32_t)e & (n - 1)]; };
    const uint32_t fac = scale ? (uint32_t)modinv(n % q, modulus) : 1u;
    out.assign((size_t)tc_words(M.LK) * 4, 0);
    uint32_t* A = out.data();
    uint32_t* B = A + (size_t)tc_a_words(M.LK) * 4;
    uint32_t* W = B + (size_t)tc_b_words(M.LK) * 4;
    // the index maps of all columns and rows once
    int cp[32], cc[32], mr[16];
    for (int i = 0; i < 8 * NT; ++i) M.col(i >> 3, i & 7, &cp[i], &cc[i]);
    for (int i = 0; i < 16; ++i) mr[i] = M.m(i);
    // a matrix entry's limbs, from its exponent: of 256 w and of w
    struct Pair {
        Limbs hi, lo;
    };
    std::vector<Pair> la(n), lb(n);
    for (uint32_t e = 0; e < n; ++e) {
        const uint32_t w = pw[e], w256 = w * 256 % q;
        if (e % M.R2 == 0) la[e] = {limbs(w256, q, 2), limbs(w, q, 2)};
        if (e % M.R1 == 0) lb[e] = {limbs(w256, q, 512), limbs(w, q, 512)};
    }
    const Limbs zero = {0, 0};
    for (int lane = 0; lane < 32; ++lane) {
        const int g = lane >> 2, t = lane & 3;
        // stage 1, A operand: h(256 W), h(W), l(256 W), l(W)
        for (int s = 0; s < S1; ++s)
            for (int r = 0; r < 4; ++r) {
                const int row = g + 8 * (r & 1), k0 = 2 * t + 8 * (r >> 1);
                Limbs hi[2], lo[2];
                for (int e = 0; e < 2; ++e) {
                    const Pair& x = la[(uint32_t)(mr[row] * M.u(s, k0 + e) * M.R2) & (n - 1)];
                    hi[e] = x.hi;
                    lo[e] = x.lo;
                }
                const uint32_t word[4] = {hi[0].h | hi[1].h << 16, lo[0].h | lo[1].h << 16, hi[0].l | hi[1].l << 16,
                                          lo[0].l | lo[1].l << 16};
                for (int i = 0; i < 4; ++i) A[((s * 4 + i) * 32 + lane) * 4 + r] = word[i];
            }
        // stage 2, B operand: {256 h(256 V) pairs 0 1, 256 h(V) pairs 0 1}, the same of l
        for (int s = 0; s < S2; ++s)
            for (int jj = 0; jj < 2; ++jj) {
                int po, v;
                M.out(jj, g, &po, &v);
                for (int r = 0; r < 2; ++r) {
                    Limbs hi[2], lo[2];
                    for (int e = 0; e < 2; ++e) {
                        const int k = 16 * s + 2 * t + 8 * r + e;
                        const Pair& x = lb[(uint32_t)(cc[k] * v * M.R1) & (n - 1)];
                        hi[e] = cp[k] == po ? x.hi : zero;
                        lo[e] = cp[k] == po ? x.lo : zero;
                    }
                    uint32_t* h = B + (((s * 2 + jj) * 2 + 0) * 32 + lane) * 4;
                    uint32_t* l = B + (((s * 2 + jj) * 2 + 1) * 32 + lane) * 4;
                    h[r] = hi[0].h | hi[1].h << 16;
                    h[2 + r] = lo[0].h | lo[1].h << 16;
                    l[r] = hi[0].l | hi[1].l << 16;
                    l[2 + r] = lo[0].l | lo[1].l << 16;
                }
            }
        // twiddles root^(m c) (times n^-1 for a scaled inverse), Shoup pairs
        for (int j = 0; j < NT; ++j)
            for (int p = 0; p < S1; ++p)
                for (int i = 0; i < 4; ++i) {
                    const int c = cc[8 * j + 2 * t + (i & 1)], m = mr[g + 8 * (i >> 1)] + 16 * p;
                    const uint32_t w = power(m * c) * fac % q;
                    uint32_t* d = W + (((j * S1 + p) * 2 + (i >> 1)) * 32 + lane) * 4 + 2 * (i & 1);
                    const uint32_t hi = (w << 16) / q;
                    d[0] = w;
                    d[1] = hi << 16 | ((w << 16) % q << 16) / q;      // floor(w 2^32 / q)
                }
    }
    *ke = ((1u << 28) / q) * q;
    *corr = (q - (32768u * 16) % q) % q;
}

}  // namespace gbntt
