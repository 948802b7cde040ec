// tc_tables.h -- shapes and host-built tables of the tensor-core transforms
// (tc16.cuh).
#pragma once

#include <cstdint>
#include <vector>

namespace gbntt {

// ---------------------------------------------------------------------------
// shapes: LK = 8 (n = 2^5 .. 2^8: 256 / n polynomials side by side, the
// stage-2 matrix block diagonal), 9 or 10
// ---------------------------------------------------------------------------
constexpr int TC_MIN_L = 5, TC_MAX_L = 10;
constexpr int tc_lk(int L) { return L <= 8 ? 8 : L; }
constexpr int tc_r1(int LK) { return LK == 10 ? 32 : 16; }
constexpr int tc_cols(int LK) { return LK == 8 ? 16 : 32; }   // stage-2 columns of a unit
constexpr int tc_s1(int LK) { return tc_r1(LK) / 16; }       // even/odd sets of stage 1
constexpr int tc_s2(int LK) { return tc_cols(LK) / 16; }     // and of stage 2
constexpr int tc_unit_coefs(int LK) { return tc_r1(LK) * tc_cols(LK); }
constexpr int TC_TILE = 1024;                       // coefficients a warp transforms per step
// table layout, in 16-byte words: stage-1 A fragments [set][4][lane], stage-2
// B fragments [set][2][2][lane], twiddle pairs [n-tile][m-tile][2][lane]
constexpr int tc_a_words(int LK) { return tc_s1(LK) * 4 * 32; }
constexpr int tc_b_words(int LK) { return tc_s2(LK) * 4 * 32; }
constexpr int tc_tw_words(int LK) { return (tc_cols(LK) / 8) * tc_s1(LK) * 2 * 32; }
constexpr int tc_words(int LK) { return tc_a_words(LK) + tc_b_words(LK) + tc_tw_words(LK); }

// a canonical int16 transform of 2^L coefficients modulo q has a tensor-core form
bool tc_supported(int L, int64_t q);
// its table (32-bit words, uploaded as it is); ke: the multiple of q just below
// 2^28 that keeps the sums non-negative; corr: -2^19 mod q, the constant that
// 16 inputs shifted by 2^15 add to the row m = 0
void tc_build(int L, int64_t q, int64_t root, bool inverse, bool natural, bool scale, std::vector<uint32_t>& out,
              uint32_t* ke, uint32_t* corr);

}  // namespace gbntt
