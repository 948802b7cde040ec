// tc16.cuh -- canonical int16 transforms of 2^5 .. 2^10 coefficients on the
// tensor cores (families F_C16F and F_C16I).
//
// A transform of n = R1 R2 coefficients is two short dense DFTs with one
// twiddle multiplication between them: with the natural input index
// R2 u + c and the natural output index m + R1 v,
//     Y[m][c] = sum_u w1^(u m) x[u][c]                    w1 = root^R2  (stage 1)
//     Z[m][v] = sum_c w2^(c v) root^(m c) Y[m][c]         w2 = root^R1  (stage 2)
// Both sums are matrix products, so they run on mma.sync.m16n8k16 (fp16
// operands, fp32 accumulation).  The accumulator layout of one mma is the A
// operand layout of the next, so a polynomial stays in the registers of one
// warp from load to store: no exchange buffer, no barrier of several warps.
//
// Exactness.  Every value is a small integer in units of 2^-23:
//   * data: a 16-bit unsigned value is split into two bytes; a byte b in a
//     16-bit lane is the fp16 subnormal b 2^-24, so the split costs a mask or
//     a byte permutation and no conversion;
//   * matrices: W and 256 W mod q (for the low and the high byte), each
//     centred and split as 256 h + l into two fp16 integers (times 2);
//   * the sums of h and of l products stay below 16 x 2 x 255 x 128 < 2^20.1
//     units each, so every partial sum is exact in fp32.  Started at 1.5
//     (whose unit in the last place is 2^-23) the sum can be read off the low
//     mantissa bits, which needs no conversion either.
//   * a 32-point DFT is two 16-point ones over the even and the odd inputs
//     (the factor w^m of the odd ones folded into their matrix), then the sum
//     and the difference: half the products of the 32-point matrix.
// Stage 1 joins 256 H + L in integers and multiplies by the twiddle with
// Shoup's method (device.cuh), which leaves [0, 2q).  Stage 2 reduces in
// floating point: its matrix carries 256 h, so H + L is the value, and H + L
// - q rint((H + L) / q) is exact term by term (H - c q, then + L).  The high
// half of a 32 x 32-bit product shares its issue slots with mma.sync on this
// part (one of each: 14.6 clocks a warp against 8 and 4 alone), so a reduction
// without it pays where no twiddle is needed.
// The factor n^-1 of a scaled inverse is folded into the twiddles, bit
// reversals into the matrices' row and column orders and the addresses.
//
// Raw int16 inputs enter as x + 2^15 (the sign bit flipped); the constant's
// transform is 2^15 R1 at m = 0 and 0 elsewhere, and is taken off there.
//
// What bounds it: 64 multiply-adds per coefficient and stage run at the
// measured 1024 per clock and SM, 16 of the 40 clocks that a warp's 32
// coefficients take per scheduler; the rest is the mma's hold on the issue
// port.  Measured, 2^26 coefficients (bytes read and written):
// n = 256 3.5 TB/s, 512 3.1-3.3, 1024 3.1-3.2; the window/exchange kernel of
// device.cuh 2.4, 2.2 and 2.0.  Sums all in integers (two high products per
// coefficient) 3.0-3.3 TB/s, all in floating point 2.6-3.3; inputs loaded to
// registers one step ahead instead of the shared-memory ring 2.5-3.0; 3 or 5
// CTAs per SM instead of 4 within 10 % below; two polynomials of 1024 points
// side by side (tables read once for both) 2.9-3.1.
#pragma once

#include "persist.cuh"
#include "tc_tables.h"

namespace gbntt {

// 128-thread CTAs, four per SM: 16 warps at 128 registers a thread
constexpr int TC_CTA = 128, TC_OCC = 4;
// each warp's input ring: TC_RING steps of TC_TILE coefficients, filled
// TC_RING - 1 steps ahead
constexpr int TC_RING = 3, TC_STEP_BYTES = 2 * TC_TILE;
constexpr int TC_WARP_RING = TC_RING * TC_STEP_BYTES;

constexpr unsigned TC_ONE5 = 0x3FC00000u;           // 1.5f
constexpr unsigned TC_CANCEL = 16384u;              // 256 (1.5f + TC_CANCEL) + 1.5f = 0 mod 2^32 on the raw bits
constexpr unsigned TC_LOW = 0x00FF00FFu;            // low bytes of both 16-bit halves

__device__ __forceinline__ void tc_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                       unsigned b1, float c0, float c1, float c2, float c3) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// high bytes of both halves as 16-bit lanes
__device__ __forceinline__ unsigned tc_high(unsigned w) { return __byte_perm(w, 0, 0x4341); }

// a constant the compiler keeps in its register instead of moving it anew
// into every mma's start quad
__device__ __forceinline__ float tc_pin(unsigned bits) {
    float f;
    asm volatile("mov.b32 %0, %1;" : "=f"(f) : "r"(bits));
    return f;
}

// The scalars of one segment.  Stage 1 of two sets starts every accumulator at
// 1.5 and takes the constants off in the addition that joins the sets; of one
// set it starts at values that leave 256 H + L + ke.  ke is a multiple of q
// just below 2^28, above every sum's magnitude (8160 q at most).
struct TcConst {
    unsigned q, q2, ke;       // q2: q in both 16-bit halves
    unsigned sum, sum0;       // added to even + odd: ke less the starts; sum0: in the row m = 0
    float h, l, l0;           // starts of a one-set stage 1; l0: the row m = 0
    float s0, s1, s2, s3;     // the quad of 1.5
    float k, qs, m;           // stage 2: 2^23 / q, q 2^-23, and 1.5 2^23 less the start's 1.5 k
};

__device__ __forceinline__ TcConst tc_const(const KArgs& a, int lane) {
    TcConst c;
    c.q = (unsigned)a.q;
    c.q2 = c.q * 0x10001u;
    c.ke = (unsigned)a.tc_ke;
    const unsigned corr = lane < 4 ? (unsigned)a.tc_corr : 0u;
    c.sum = c.ke - 2u * 257u * TC_ONE5;
    c.sum0 = c.sum + 2u * corr;
    c.h = __uint_as_float(TC_ONE5 + TC_CANCEL + (c.ke >> 8));
    c.l = __uint_as_float(TC_ONE5 + (c.ke & 255u));
    c.l0 = __uint_as_float(TC_ONE5 + (c.ke & 255u) + corr);
    c.s0 = tc_pin(TC_ONE5);
    c.s1 = tc_pin(TC_ONE5);
    c.s2 = tc_pin(TC_ONE5);
    c.s3 = tc_pin(TC_ONE5);
    c.k = __fdiv_rn(8388608.f, (float)a.q);
    c.qs = (float)a.q * (1.f / 8388608.f);
    c.m = __fsub_rn(12582912.f, 1.5f * c.k);
    return c;
}

// stage 1: 256 H + L on the raw bits
__device__ __forceinline__ unsigned tc_join(float h, float l) {
    return (__float_as_uint(h) << 8) + __float_as_uint(l);
}
// stage 2: h + l less a nearby multiple of q, above -q and below q, in the low
// mantissa bits (l carries the start 1.5).  h is a multiple of 256 units below
// 2^28, l below 2^22 units, the quotient below 8161, so each operation but the
// quotient is exact; the quotient is off by less than one (tc_supported).
__device__ __forceinline__ unsigned tc_reduce(float h, float l, const TcConst& k) {
    const float c = __fsub_rn(__fmaf_rn(__fadd_rn(h, l), k.k, k.m), 12582912.f);
    return __float_as_uint(__fadd_rn(__fmaf_rn(c, -k.qs, h), l));
}
// two of them as residues in [0, q), in 16-bit halves
__device__ __forceinline__ unsigned tc_pack(unsigned a, unsigned b, unsigned q2) {
    const unsigned t = __byte_perm(a, b, 0x5410);
    return __viaddmin_u16x2(t, q2, t);                // a negative t is above t + q as an unsigned half
}

// A table load the compiler must not keep in registers across steps (the
// tables stay in L1; a step re-reads them).
__device__ __forceinline__ uint4 tc_tab(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
// one lane's share of a step's input, copied asynchronously into the warp's
// buffer in 16-byte pieces (bytes: what the segment still holds)
__device__ __forceinline__ void tc_fetch(unsigned char* dst, const short* src, int bytes, int lane) {
#pragma unroll
    for (int i = 0; i < TC_STEP_BYTES / 512; ++i) {
        const int o = 512 * i + 16 * lane;
        if (o < bytes)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst + o)),
                         "l"(reinterpret_cast<const char*>(src) + o)
                         : "memory");
    }
}
__device__ __forceinline__ void tc_fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tc_fetch_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// raw input words of one unit
template <int LK>
struct TcRaw {
    unsigned w[tc_unit_coefs(LK) / 64];
};

// LB: bit-reversed input (pairs of rows are adjacent), else natural.  base: the
// unit's first coefficient in the staged step; l2: log2 R2
template <int LK, bool LB>
__device__ __forceinline__ void tc_load(TcRaw<LK>& r, const short* base, int lane, int l2) {
    const int g = lane >> 2, t = lane & 3;
    constexpr int S1 = tc_s1(LK), NT = tc_cols(LK) / 8, R1 = tc_r1(LK);
    if constexpr (LB) {
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int s = 0; s < S1; ++s) {
                const uint2 v = *reinterpret_cast<const uint2*>(base + R1 * (8 * j + g) + 16 * s + 4 * t);
                r.w[(j * S1 + s) * 2] = v.x;
                r.w[(j * S1 + s) * 2 + 1] = v.y;
            }
    } else if constexpr (LK == 8) {
        const int R2m = (1 << l2) - 1, c = 2 * g;
        const int b0 = ((c >> l2) << (4 + l2)) + (c & R2m);
#pragma unroll
        for (int e = 0; e < 4; ++e)
            r.w[e] = *reinterpret_cast<const unsigned*>(base + b0 + ((2 * t + (e & 1) + 8 * (e >> 1)) << l2));
    } else {
#pragma unroll
        for (int s = 0; s < S1; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = 2 * t + (e & 1) + 8 * (e >> 1);
                const uint2 v = *reinterpret_cast<const uint2*>(base + (S1 * k + s) * 32 + 4 * g);
                r.w[(s * 4 + e) * 2] = v.x;
                r.w[(s * 4 + e) * 2 + 1] = v.y;
            }
    }
}

// the B operand of set s, n-tile j: low- and high-byte lanes, k pairs 0 and 1
template <int LK, bool LB>
__device__ __forceinline__ void tc_fields(const TcRaw<LK>& r, int s, int j, unsigned (&lo)[2], unsigned (&hi)[2]) {
    constexpr int S1 = tc_s1(LK);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if constexpr (LB) {
            const unsigned w = r.w[(j * S1 + s) * 2 + h];
            lo[h] = w & TC_LOW;
            hi[h] = tc_high(w ^ 0x80008000u);
        } else {
            // words of the two rows of the pair that hold this tile's column
            const bool wide = LK > 8;
            const unsigned a = wide ? r.w[(s * 4 + 2 * h) * 2 + (j & 1)] : r.w[2 * h];
            const unsigned b = wide ? r.w[(s * 4 + 2 * h + 1) * 2 + (j & 1)] : r.w[2 * h + 1];
            const bool upper = wide ? j >> 1 : j;
            lo[h] = __byte_perm(a & TC_LOW, b & TC_LOW, upper ? 0x7632 : 0x5410);
            hi[h] = __byte_perm((a & ~TC_LOW) ^ 0x80008000u, (b & ~TC_LOW) ^ 0x80008000u, upper ? 0x6723 : 0x4501);
        }
    }
}

// stores rows g and g + 8 of m-tile p.  Z[d][jj][i]: d = 0 the sum, d = 1 the
// difference (outputs v and v + 16); SB: bit-reversed output, else natural;
// FULL: the whole unit lies in the segment, else avail coefficients of it do
template <int LK, bool SB, bool FULL>
__device__ __forceinline__ void tc_store(const unsigned (&Z)[tc_s2(LK)][2][4], int p, short* __restrict__ base,
                                         int avail, int lane, int l2, unsigned q2) {
    constexpr int S1 = tc_s1(LK), S2 = tc_s2(LK), R1 = tc_r1(LK);
    const int g = lane >> 2, t = lane & 3;
    if constexpr (SB) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = S1 == 2 ? 2 * (g + 8 * h) + p : g + 8 * h;
            if constexpr (S2 == 2) {
                uint4 o;
                o.x = tc_pack(Z[0][0][2 * h], Z[1][0][2 * h], q2);
                o.y = tc_pack(Z[0][0][2 * h + 1], Z[1][0][2 * h + 1], q2);
                o.z = tc_pack(Z[0][1][2 * h], Z[1][1][2 * h], q2);
                o.w = tc_pack(Z[0][1][2 * h + 1], Z[1][1][2 * h + 1], q2);
                *reinterpret_cast<uint4*>(base + row * 32 + 8 * t) = o;
            } else {
                const unsigned o0 = tc_pack(Z[0][0][2 * h], Z[0][0][2 * h + 1], q2);
                const unsigned o1 = tc_pack(Z[0][1][2 * h], Z[0][1][2 * h + 1], q2);
                const int c = 4 * t, R2m = (1 << l2) - 1;
                const int pos = ((c >> l2) << (4 + l2)) + (c & R2m) + (row << l2);
                if (l2 >= 2) {
                    if (FULL || pos < avail) *reinterpret_cast<uint2*>(base + pos) = make_uint2(o0, o1);
                } else {                        // n = 32: two polynomials
                    if (FULL || pos < avail) *reinterpret_cast<unsigned*>(base + pos) = o0;
                    if (FULL || pos + 32 < avail) *reinterpret_cast<unsigned*>(base + pos + 32) = o1;
                }
            }
        }
    } else {
#pragma unroll
        for (int d = 0; d < S2; ++d)
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const unsigned o = tc_pack(Z[d][jj][e], Z[d][jj][2 + e], q2);
                    const int pos = R1 * (8 * jj + 2 * t + e + 16 * d) + 2 * g + 16 * p;
                    if (FULL || pos < avail) *reinterpret_cast<unsigned*>(base + pos) = o;
                }
    }
}

// One step: the TC_TILE / tc_unit_coefs(LK) units of a tile together, so that
// each table word is read once for all of them and their instruction streams
// overlap.  in: the staged tile (what lies past avail coefficients is transformed
// with it and not stored)
template <int LK, bool LB, bool SB>
__device__ __forceinline__ void tc_step(const short* in, short* __restrict__ out, int avail, int lane, int l2,
                                        const uint4* __restrict__ tab, const TcConst& k) {
    constexpr int S1 = tc_s1(LK), S2 = tc_s2(LK), NT = tc_cols(LK) / 8, UC = tc_unit_coefs(LK), U = TC_TILE / UC;
    const bool full = avail == TC_TILE;
    TcRaw<LK> raw[U];
#pragma unroll
    for (int u = 0; u < U; ++u) tc_load<LK, LB>(raw[u], in + u * UC, lane, l2);
    unsigned P[U][S1][NT][2];       // twiddled stage-1 results below 2q, two columns per word
    {
        uint4 A[S1][4];
#pragma unroll
        for (int s = 0; s < S1; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) A[s][i] = tc_tab(tab + (s * 4 + i) * 32);
        const uint4* tw = tab + tc_a_words(LK) + tc_b_words(LK);
#pragma unroll
        for (int jo = 0; jo < NT; ++jo) {
            const int j = NT == 4 ? ((jo & 1) << 1) | (jo >> 1) : jo;   // tiles that share input words in turn
            uint4 w[S1][2];
#pragma unroll
            for (int p = 0; p < S1; ++p)
#pragma unroll
                for (int i = 0; i < 2; ++i) w[p][i] = tc_tab(tw + ((j * S1 + p) * 2 + i) * 32);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                unsigned T[S1][4];
#pragma unroll
                for (int s = 0; s < S1; ++s) {
                    unsigned lo[2], hi[2];
                    tc_fields<LK, LB>(raw[u], s, j, lo, hi);
                    float H[4], Lo[4];
                    tc_mma(H, A[s][0].x, A[s][0].y, A[s][0].z, A[s][0].w, hi[0], hi[1], S1 == 2 ? k.s0 : k.h,
                           S1 == 2 ? k.s1 : k.h, S1 == 2 ? k.s2 : k.h, S1 == 2 ? k.s3 : k.h);
                    tc_mma(Lo, A[s][2].x, A[s][2].y, A[s][2].z, A[s][2].w, hi[0], hi[1], S1 == 2 ? k.s0 : k.l0,
                           S1 == 2 ? k.s1 : k.l0, S1 == 2 ? k.s2 : k.l, S1 == 2 ? k.s3 : k.l);
                    tc_mma(H, A[s][1].x, A[s][1].y, A[s][1].z, A[s][1].w, lo[0], lo[1], H[0], H[1], H[2], H[3]);
                    tc_mma(Lo, A[s][3].x, A[s][3].y, A[s][3].z, A[s][3].w, lo[0], lo[1], Lo[0], Lo[1], Lo[2], Lo[3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) T[s][i] = tc_join(H[i], Lo[i]);
                }
#pragma unroll
                for (int p = 0; p < S1; ++p) {
                    unsigned y[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if constexpr (S1 == 2)
                            y[i] = p ? T[0][i] - T[1][i] + k.ke : T[0][i] + T[1][i] + (i < 2 ? k.sum0 : k.sum);
                        else
                            y[i] = T[0][i];
                    }
                    const unsigned r0 = shoup_mul(y[0], w[p][0].x, w[p][0].y, k.q);
                    const unsigned r1 = shoup_mul(y[1], w[p][0].z, w[p][0].w, k.q);
                    const unsigned r2 = shoup_mul(y[2], w[p][1].x, w[p][1].y, k.q);
                    const unsigned r3 = shoup_mul(y[3], w[p][1].z, w[p][1].w, k.q);
                    P[u][p][j][0] = __byte_perm(r0, r1, 0x5410);
                    P[u][p][j][1] = __byte_perm(r2, r3, 0x5410);
                }
            }
        }
    }
    uint4 B[S2][2][2];
#pragma unroll
    for (int s = 0; s < S2; ++s)
#pragma unroll
        for (int i = 0; i < 4; ++i) B[s][i >> 1][i & 1] = tc_tab(tab + tc_a_words(LK) + (s * 4 + i) * 32);
#pragma unroll
    for (int p = 0; p < S1; ++p)
#pragma unroll
        for (int u = 0; u < U; ++u) {
            float H[S2][2][4], Lo[S2][2][4];
#pragma unroll
            for (int s = 0; s < S2; ++s) {
                const unsigned w[4] = {P[u][p][2 * s][0], P[u][p][2 * s][1], P[u][p][2 * s + 1][0],
                                       P[u][p][2 * s + 1][1]};
                const unsigned lo[4] = {w[0] & TC_LOW, w[1] & TC_LOW, w[2] & TC_LOW, w[3] & TC_LOW};
                const unsigned hi[4] = {tc_high(w[0]), tc_high(w[1]), tc_high(w[2]), tc_high(w[3])};
#pragma unroll
                for (int jj = 0; jj < 2; ++jj) {
                    float (&h)[4] = H[s][jj];
                    float (&l)[4] = Lo[s][jj];
                    const uint4 bh = B[s][jj][0], bl = B[s][jj][1];
                    tc_mma(h, hi[0], hi[1], hi[2], hi[3], bh.x, bh.y, 0.f, 0.f, 0.f, 0.f);
                    tc_mma(l, hi[0], hi[1], hi[2], hi[3], bl.x, bl.y, s ? 0.f : k.s0, s ? 0.f : k.s1,
                           s ? 0.f : k.s2, s ? 0.f : k.s3);
                    tc_mma(h, lo[0], lo[1], lo[2], lo[3], bh.z, bh.w, h[0], h[1], h[2], h[3]);
                    tc_mma(l, lo[0], lo[1], lo[2], lo[3], bl.z, bl.w, l[0], l[1], l[2], l[3]);
                }
            }
            unsigned Z[S2][2][4];
#pragma unroll
            for (int jj = 0; jj < 2; ++jj)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if constexpr (S2 == 2) {
                        Z[0][jj][i] = tc_reduce(H[0][jj][i] + H[1][jj][i], Lo[0][jj][i] + Lo[1][jj][i], k);
                        Z[1][jj][i] = tc_reduce(H[0][jj][i] - H[1][jj][i], Lo[0][jj][i] - Lo[1][jj][i], k);
                    } else {
                        Z[0][jj][i] = tc_reduce(H[0][jj][i], Lo[0][jj][i], k);
                    }
                }
            if (full) tc_store<LK, SB, true>(Z, p, out + u * UC, UC, lane, l2, k.q2);
            else if (LK == 8) tc_store<LK, SB, false>(Z, p, out + u * UC, avail - u * UC, lane, l2, k.q2);
            else if (u * UC < avail) tc_store<LK, SB, true>(Z, p, out + u * UC, UC, lane, l2, k.q2);
        }
}

// the tiles first, first + step, ... below last of one segment (a tile =
// TC_TILE coefficients), by one warp; ring: the warp's TC_WARP_RING bytes of
// shared memory
template <int LK, bool LB, bool SB>
__device__ __forceinline__ void tc_segment(const KArgs& a, int L, long long first, long long last, long long step,
                                           int lane, unsigned char* ring) {
    const short* __restrict__ in = static_cast<const short*>(a.in);
    short* __restrict__ out = static_cast<short*>(a.out);
    const long long total = a.batch << L;
    const uint4* tab = a.tctab + lane;
    auto rest = [&](long long tile) {                     // coefficients of the tile
        const long long r = total - tile * TC_TILE;
        return r < TC_TILE ? (int)r : TC_TILE;
    };
    auto fetch = [&](long long tile, int slot) {
        if (tile < last) tc_fetch(ring + slot * TC_STEP_BYTES, in + tile * TC_TILE, 2 * rest(tile), lane);
        tc_fetch_commit();
    };
    __syncwarp();                                         // the ring's previous use is over
    long long ahead = first;
#pragma unroll
    for (int i = 0; i < TC_RING - 1; ++i) {
        fetch(ahead, i);
        ahead += step;
    }
    const TcConst k = tc_const(a, lane);
    int slot = 0;
    for (long long tile = first; tile < last; tile += step) {
        tc_fetch_wait<TC_RING - 2>();
        __syncwarp();                      // every lane's pieces of this step are there, and the previous step is read
        fetch(ahead, slot == 0 ? TC_RING - 1 : slot - 1);
        ahead += step;
        tc_step<LK, LB, SB>(reinterpret_cast<const short*>(ring + slot * TC_STEP_BYTES), out + tile * TC_TILE,
                            rest(tile), lane, L - 4, tab, k);
        slot = slot + 1 == TC_RING ? 0 : slot + 1;
    }
    tc_fetch_wait<0>();
}

}  // namespace gbntt
