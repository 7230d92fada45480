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
PT_HD float EnvRow(float r, int H) {
    const float x = r * (float)H - 1.0f;
    const float k = floorf(x);
    const float y = x > 0.0f && x == k ? x : fmaxf(k, 0.0f) + 0.5f;
    return y * (1.0f / (float)H);
}

}  // namespace ptg
