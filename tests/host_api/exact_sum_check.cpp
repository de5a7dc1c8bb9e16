// exact_sum.h against 128-bit integer sums: sets of up to 256 floats, "near" within
// 2^32 of the largest (the sum is exact and rounded once) and "far" (bits below
// 2^-55 of the largest go), and the edges: zeros, the largest floats, the smallest
// normal ones, single terms.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "exact_sum.h"

static uint32_t bits(float x) {
    uint32_t u;
    std::memcpy(&u, &x, 4);
    return u;
}

// The sum in units of 2^(low - 150) for terms with exponent fields in [low, low + 90].
static unsigned __int128 exact(const std::vector<float>& x, int low) {
    unsigned __int128 s = 0;
    for (float v : x)
        if (v != 0.0f) s += (unsigned __int128)((bits(v) & 0x7FFFFFu) | 0x800000u) << ((int)(bits(v) >> 23) - low);
    return s;
}

int main() {
    std::mt19937 rng(7);
    int bad = 0, sets = 0;
    auto check = [&](const std::vector<float>& x, int low, double terms_lost) {
        uint32_t top = 0;
        for (float v : x) top = std::max(top, bits(v) >> 23);
        uint64_t s = 0;
        for (float v : x) s += mcd::fixed_term(bits(v), top);
        const double got = mcd::fixed_value(s, top);
        // Half an ulp of the sum, plus a unit for each term that may lose bits.
        const long double unit = std::ldexp(1.0L, low - 150);
        const unsigned __int128 e = exact(x, low);
        const long double hi = (long double)(uint64_t)(e >> 64) * 18446744073709551616.0L + (long double)(uint64_t)e;
        const unsigned __int128 g = (unsigned __int128)std::ldexp(got, 150 - low);
        const unsigned __int128 err = g > e ? g - e : e - g;
        const long double allowed = hi * std::ldexp(1.0L, -53) + terms_lost * std::ldexp(1.0L, (int)top - 182) / unit;
        sets++;
        if ((long double)err > allowed) bad++;
    };
    for (int n : {1, 2, 63, 64, 128, 256})
        for (int t = 0; t < 2000; t++) {
            const int low = 1 + (int)(rng() % 150);
            std::vector<float> near, far;
            for (int k = 0; k < n; k++) {
                const float m = 1.0f + (float)(rng() & 0x7FFFFF) / 8388608.0f;
                near.push_back(rng() % 9 ? std::ldexp(m, low - 127 + (int)(rng() % 33)) : 0.0f);
                far.push_back(std::ldexp(m, low - 127 + (int)(rng() % 64)));
            }
            check(near, low, 0);
            check(far, low, n);
        }
    check({0.0f, 0.0f}, 1, 0);
    check({std::ldexp(1.0f, -126)}, 1, 0);
    check(std::vector<float>(256, 3.4028235e38f), 254 - 60, 0);
    std::printf("SETS %d BAD %d\n", sets, bad);
    return bad != 0;
}
