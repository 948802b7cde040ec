// Host-side check of the lane rounding of the staged batch kernel against the
// other kernels' (device.cuh): constructed ties, extremes and random pairs.
#include <cstdint>
#include <cstdio>

#include "../../ntts_on_amd_ai_engines_aie1_gb300/csrc/device.cuh"

int main() {
    uint64_t state = 0x9E3779B97F4A7C15ull, checked = 0, bad = 0;
    auto rnd = [&] { return (uint32_t)((state = state * 6364136223846793005ull + 1442695040888963407ull) >> 32); };
    auto check = [&](int32_t a, int32_t b) {
        ++checked;
        if (gbntt::rsz32p(a, b) != gbntt::rsz32(a, b) && bad++ < 10) std::printf("rsz32p: %d %d\n", a, b);
        const int q = 998244353;
        if (gbntt::br32<gbntt::FORM_STAGED>(a, b, q) != gbntt::br32(a, b, q) ||
            gbntt::bm32<gbntt::FORM_STAGED>(a, b ^ 5, b, q) != gbntt::bm32(a, b ^ 5, b, q))
            if (bad++ < 10) std::printf("products: %d %d\n", a, b);
    };
    const int32_t edge[] = {0, 1, -1, 2, -2, INT32_MIN, INT32_MIN + 1, INT32_MAX, 1 << 30, -(1 << 30), 3 << 29, 65536, -65536};
    for (int32_t a : edge)
        for (int32_t b : edge) check(a, b);
    for (int z = 0; z < 31; ++z)
        for (int i = 0; i < 2000; ++i) {
            const int32_t b = (int32_t)((rnd() | 1u) << z), a = (int32_t)((rnd() | 1u) << (31 - z));   // a b = 2^31 mod 2^32
            check(a, b);
            check(-a, b);
            check(b, a);
        }
    for (int i = 0; i < 4000000; ++i) check((int32_t)rnd(), (int32_t)rnd());
    std::printf("%llu pairs checked, %llu failures\n", (unsigned long long)checked, (unsigned long long)bad);
    return bad ? 1 : 0;
}
