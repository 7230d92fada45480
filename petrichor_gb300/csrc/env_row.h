// Row of the environment sampler for maps whose height is a power of two, in plain float
// arithmetic that also compiles for the host (tests/cpp/env_row.cpp compares it with the
// search it replaces).
#pragma once
#include <cmath>

#include "pt_layout.h"

namespace ptg {

// The reference bisects [0, 1) for the row coordinate v until the interval is one row (1 / H)
// wide and takes its middle, comparing v + 1 / H with r at every midpoint v (the tables it
// searches are that function of v alone, EnvSample); a midpoint that compares equal ends the
// search there. The midpoints are multiples of 1 / H, so with x = r H - 1 (exact: a power of
// two times r, less one) the search ends at x / H when x is a whole number above 0 and in the
// middle of row max(floor(x), 0) otherwise. One expression took the place of log2 H
// dependent steps in the shade stage and the replay.
//
// EnvRowAt: v H, a multiple of 1/2 in [1/2, H).
PT_HD float EnvRowAt(float r, int H) {
    const float x = r * (float)H - 1.0f;
    const float k = floorf(x);
    return x > 0.0f && x == k ? x : fmaxf(k, 0.0f) + 0.5f;
}
PT_HD float EnvRow(float r, int H) { return EnvRowAt(r, H) * (1.0f / (float)H); }

// The column is the same for every draw (EnvSample), so a scene's sampler has 2 H outcomes at
// most: direction and radiance of each are kept in a table for maps of up to this many rows
// (2 H entries of 32 bytes: 64 KB at 1024 rows, 512 KB here).
constexpr int kEnvTableRows = 8192;

}  // namespace ptg
