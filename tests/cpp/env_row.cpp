// EnvRow (csrc/env_row.h) against the bisection it replaces: every 24-bit uniform draw for a
// few heights, and for every height up to 2^22 a spread of draws, all rows' exact borders and
// their neighbours, draws with more bits (u / 2^32 as the reference forms them), 0 and 1.
// Prints "ok <cases>" or the first difference.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "env_row.h"

static float Search(float r0, int H) {
    const float th = 1.0f / (float)H;
    float v0 = 0.0f, v1 = 1.0f;
    for (int it = 0; it < 64; it++) {
        const float v = 0.5f * (v0 + v1);
        const float diff = (v + th) - r0;
        if (v1 - v0 <= th) return v;
        if (diff > 0) v1 = v;
        else if (diff < 0) v0 = v;
        else return v;
    }
    return v0;
}

int main() {
    long cases = 0;
    auto check = [&](float r, int H) {
        cases++;
        const float a = ptg::EnvRow(r, H), b = Search(r, H);
        if (a == b) return true;
        std::printf("differs: r %.9g H %d: %.9g, search %.9g\n", r, H, a, b);
        return false;
    };
    for (int H : {1, 2, 512, 4096})
        for (uint32_t m = 0; m < (1u << 24); m++)
            if (!check((float)m * (1.0f / 16777216.0f), H)) return 1;
    uint64_t s = 1;
    auto next = [&] {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (uint32_t)(s >> 32);
    };
    for (int h = 0; h <= 22; h++) {
        const int H = 1 << h;
        const long rows = H < 4096 ? H : 4096;
        for (long k = 0; k <= rows; k++) {
            const float b = (float)(H < 4096 ? k : (next() % (uint32_t)H)) / (float)H;
            if (!check(b, H) || !check(std::nextafterf(b, 0.0f), H) || !check(fminf(std::nextafterf(b, 2.0f), 1.0f), H))
                return 1;
        }
        for (int k = 0; k < 200000; k++) {
            const uint32_t u = next();
            if (!check((float)(u >> 8) * (1.0f / 16777216.0f), H)) return 1;
            if (!check((float)u / 4294967296.0f, H)) return 1;
            if (!check((float)(u >> (u & 31)) / 4294967296.0f, H)) return 1;
        }
        if (!check(0.0f, H) || !check(1.0f, H)) return 1;
    }
    std::printf("ok %ld\n", cases);
    return 0;
}
