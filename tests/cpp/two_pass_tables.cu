// Host-side check of the tables of the canonical two-pass transforms
// (canon_tables.h): every entry that the passes read lies inside them and is
// the block that the butterfly needs, and every word has one writer.
#include <cstdio>
#include <vector>

#include "../../ntts_on_amd_ai_engines_aie1_gb300/csrc/canon_tables.h"
#include "../../ntts_on_amd_ai_engines_aie1_gb300/csrc/device.cuh"

using namespace gbntt;

static long long checked = 0, bad = 0;
static void check(bool ok, const char* what, int fam, int L, int L2, long long v) {
    ++checked;
    if (!ok && bad++ < 10) std::printf("%s: fam %d L %d L2 %d value %lld\n", what, fam, L, L2, v);
}

template <int FAM>
void rows(int L, int L2) {
    const int EL = 4, G = 1 << (L2 - EL), n1 = 1 << (L - L2);
    const long long tail = (long long)two_pass_entries(L, EL) - (long long)two_pass_blocks(L);   // in entries
    for (int r : {0, 1, n1 / 2 + 1, n1 - 1})
        for (int s = 0; s < L2; ++s) {
            const int B = step_b(FAM, L2, s), LO = window_lo(FAM, L2, EL, s);
            const int NV = step_vec_pairs<FAM, R2_WIDE>(LO, EL, B, true);
            for (int g = 0; g < G; ++g) {
                if (NV) {
                    const int e0 = ((r << L2) | posmap_c(LO, EL, g, 0)) >> (B + 1);
                    for (int i = 0; i < NV / 2; ++i) {
                        const long long at = two_pass_tail_at(L2, EL, r, NV / 2 - 1 + i, g);
                        check(at >= 0 && 2 * at + 1 < tail, "word outside the tail", FAM, L, L2, at);
                        check(at == two_pass_tail_at(L2, EL, r, 0, g) + (NV / 2 - 1 + i) * (long long)G, "word", FAM, L, L2, at);
                        check(two_pass_tail_block(L2, EL, r, NV / 2 - 1 + i, g) == e0 + 2 * i, "block", FAM, L, L2, e0);
                    }
                } else {
                    for (int k = 0; k < 16; ++k) {
                        const long long b = ((r << L2) | posmap_c(LO, EL, g, k)) >> (B + 1);
                        check(b < (long long)two_pass_blocks(L), "block outside the table", FAM, L, L2, b);
                    }
                }
            }
        }
}

int main() {
    for (int L = 14; L <= 22; ++L)
        for (int L2 = 10; L2 <= 12; ++L2) {
            const int EL = 4, L1 = L - L2;
            if (L1 < 2) continue;
            check(two_pass_entries(L, EL) * 8 <= (size_t)8 << L, "more than 8 bytes a coefficient", 0, L, L2,
                  (long long)two_pass_entries(L, EL));
            rows<F_C32F>(L, L2);
            rows<F_C32I>(L, L2);
            // the columns' blocks: below n1 / 2
            check((1ll << L1) / 2 <= (long long)two_pass_blocks(L), "column blocks", 0, L, L2, 1ll << L1);
            // each word of the tail is written once: those of bit 0 hold every
            // block where two_pass_tail_of finds it, the others copy theirs
            const int words = two_pass_tail_words(EL), first = (1 << (EL - 2)) - 1, G = 1 << (L2 - EL);
            std::vector<char> seen((size_t)words << (L - EL), 0);
            for (int r = 0; r < 1 << L1; ++r)
                for (int w = 0; w < words; ++w)
                    for (int g = 0; g < G; ++g) {
                        const long long at = two_pass_tail_at(L2, EL, r, w, g);
                        const int b = two_pass_tail_block(L2, EL, r, w, g);
                        check(at >= 0 && at < (long long)seen.size() && !seen[at]++, "word taken", 0, L, L2, at);
                        const long long from = two_pass_tail_of(L2, EL, b);
                        check(b >= 0 && b + 1 < 1 << (L - 1) && (b & 1) == 0, "pair of blocks", 0, L, L2, b);
                        if (w >= first) check(from == at, "home of a block", 0, L, L2, b);
                        // a copied word's home is a word of bit 0
                        else check((from / G) % words >= first && from < (long long)seen.size(), "source", 0, L, L2, b);
                    }
        }
    std::printf("%lld checks, %lld failures\n", checked, bad);
    return bad ? 1 : 0;
}
