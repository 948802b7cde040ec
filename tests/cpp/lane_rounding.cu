// Host-side check of the lane arithmetic of device.cuh against the rounding it
// stands for, round(p / 2^K) with ties toward zero written with the product's
// own sign: the int16 forms over every lane value and a spread of multipliers
// (every tie of them among the values), the int32 forms at constructed ties and
// on a pseudo-random sample; and the bound that lets the radix-2 int16
// butterflies of moduli below 2^14 leave out the int16 wrap.
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "../../ntts_on_amd_ai_engines_aie1_gb300/csrc/device.cuh"

static uint64_t checked = 0, bad = 0;
static void check(bool ok, const char* what, long long a, long long b) {
    ++checked;
    if (!ok && bad++ < 10) std::printf("%s: %lld %lld\n", what, a, b);
}
static int64_t round_zero(int64_t p, int k) {
    const int64_t half = (int64_t)1 << (k - 1), mag = (p < 0 ? -p : p);
    const int64_t m = (mag + half - 1) >> k;      // half rounds down in magnitude
    return p < 0 ? -m : m;
}

int main() {
    uint64_t state = 0x9E3779B97F4A7C15ull;
    auto rnd = [&] { return (uint32_t)((state = state * 6364136223846793005ull + 1442695040888963407ull) >> 32); };
    // int16: multipliers of every size and parity, with the Barrett constants
    for (int i = 0; i < 400; ++i) {
        const int fixed[] = {0, 1, -1, 2, 3, 4, 5, 6, 8, 9, 512, 16384, -16384, 32767, -32768, -32767};
        const int b = i < 16 ? fixed[i] : (int)(int16_t)rnd();
        for (int a = -32768; a <= 32767; ++a)
            check(gbntt::rsz16(a, b) == round_zero((int64_t)a * b, 16), "rsz16", a, b);
    }
    for (int c = 1; c < 512; c += 2)
        for (int a = -32768; a <= 32767; a += c < 32 ? 1 : 61)
            check(gbntt::br16_odd(a, c, 12289) == gbntt::br16(a, c, 12289), "br16_odd", a, c);
    // int32: products at 2^31 mod 2^32 (ties), zeros, extremes, random pairs
    const int32_t edge[] = {0, 1, -1, INT32_MIN, INT32_MAX, INT32_MIN + 1, 1 << 29, -(1 << 29), 1 << 30, -(1 << 30), 3 << 29};
    const int32_t mult[] = {0, 1, -1, 2, 4, 5, 6, 8, 16, -4, -8, 1 << 20, -(1 << 20), 1 << 30, INT32_MIN, INT32_MAX};
    for (int32_t b : mult) {
        for (int32_t a : edge) check(gbntt::rsz32(a, b) == (int32_t)round_zero((int64_t)a * b, 32), "rsz32", a, b);
        for (int i = 0; i < 4000 && b; ++i) {
            // a tie: a = t 2^(31 - z) where b = odd 2^z
            int z = 0;
            while (!((b >> z) & 1)) ++z;
            const int32_t a = (int32_t)((uint32_t)(rnd() | 1u) << (31 - z));
            check(gbntt::rsz32(a, b) == (int32_t)round_zero((int64_t)a * b, 32), "rsz32 tie", a, b);
            const int32_t h = (int32_t)((uint32_t)a >> 1);          // a tie of 2^31
            check(gbntt::rsz31(h, b) == (int32_t)round_zero((int64_t)h * b, 31), "rsz31 tie", h, b);
            check(gbntt::rsz31(-h, b) == (int32_t)round_zero((int64_t)-h * b, 31), "rsz31 tie", -h, b);
        }
    }
    for (int i = 0; i < 4000000; ++i) {
        const int32_t a = (int32_t)rnd(), b = (int32_t)rnd();
        check(gbntt::rsz32(a, b) == (int32_t)round_zero((int64_t)a * b, 32), "rsz32", a, b);
        check(gbntt::rsz31(a, b) == (int32_t)round_zero((int64_t)a * b, 31), "rsz31", a, b);
    }
    // radix-2 butterflies of the narrow moduli: every result is an int16
    for (int q : {97, 7681, 10753, 12289, 16381}) {
        const int c = (int)(65536.0 / q + 0.5);
        int worst = 0;
        for (int a = -32768; a <= 32767; ++a) {
            const int u = std::abs(gbntt::br16(a, c, q));
            worst = u > worst ? u : worst;
        }
        int worst_w = 0;
        for (int i = 0; i < 2000; ++i) {
            int tw = (int)(rnd() % q);
            if (tw > q / 2) tw -= q;
            // multipliers within 1.5 of tw 2^16 / q, as the tables have them
            const int wq = (int)(tw * 65536.0 / q) + (int)(rnd() % 3) - 1;
            for (int a = -32768; a <= 32767; a += 31) {
                const int w = std::abs(gbntt::bm16(a, tw, wq < -32768 ? -32768 : wq > 32767 ? 32767 : wq, q));
                worst_w = w > worst_w ? w : worst_w;
            }
        }
        check(worst + worst_w <= 32767, "u + w", worst, worst_w);
        check(gbntt::r2_form(q, c) == (c & 1 ? gbntt::R2_LEAN_ODD : gbntt::R2_LEAN), "form", q, c);
    }
    check(gbntt::r2_form(16384, 4) == gbntt::R2_WIDE && gbntt::r2_form(18433, 4) == gbntt::R2_WIDE, "wide", 0, 0);
    std::printf("%llu values checked, %llu failures\n", (unsigned long long)checked, (unsigned long long)bad);
    return bad ? 1 : 0;
}
