// Rays of a short ray query that each warp of the launch takes by its index, in plain
// integers that also compile for the host (tests/cpp/query_share.cpp).
#pragma once
#include "pt_layout.h"

namespace ptg {

// Warps per SM that a short query is spread over: all that are resident, so that a warp has few
// rays to diverge. Over 6 (the wave queues' spread) and over 28, incoherent rays in 300,000
// triangles: 3000 take 33 and 30 us, 15,000 69 and 64, 50,000 76 and 68; camera rays 59 and 42, 95 and
// 91, 93 and 89 us. With full warps, before there was a spread: 47, 64, 71; 66, 105, 120 us.
constexpr int kQueryWarps = 28;
// From a full warp of rays on the warps refill, from a counter: with shares of up to 31 instead
// of 16 rays, 115,000 rays take 81 instead of 82 us, camera rays in 1000 triangles 21 instead of 25.
constexpr int kMostShare = 31;

// Rays per warp of a query of n > 0 rays: warp w takes [w * share, (w + 1) * share). 0: the
// query is too long for that, and its warps fetch from a counter. The spread is at most the
// launch's own warps, so the shares cover the query whatever the grid.
inline int QueryShare(int n, int sms, int gridWarps) {
    const int most = sms * kQueryWarps;
    const int warps = most < gridWarps ? most : gridWarps;
    const int share = (n - 1) / warps + 1;
    return share <= kMostShare ? share : 0;
}

}  // namespace ptg
