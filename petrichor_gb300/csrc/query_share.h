// Rays of a short ray query that each warp of the launch takes by its index, in plain
// integers that also compile for the host (tests/cpp/query_share.cpp).
#pragma once
#include "pt_layout.h"

namespace ptg {

// Warps per SM that a short queue is spread over (figures at LanesUsed, wavefront.cu).
constexpr int kSpreadWarps = 6;
// Warps that take more than half a warp of rays refill, from a counter.
constexpr int kMostShare = 16;

// Rays per warp of a query of n > 0 rays: warp w takes [w * share, (w + 1) * share). 0: the
// query is too long for that, and its warps fetch from a counter. The spread is at most the
// launch's own warps, so the shares cover the query whatever the grid.
inline int QueryShare(int n, int sms, int gridWarps) {
    const int most = sms * kSpreadWarps;
    const int warps = most < gridWarps ? most : gridWarps;
    const int share = (n - 1) / warps + 1;
    return share <= kMostShare ? share : 0;
}

}  // namespace ptg
