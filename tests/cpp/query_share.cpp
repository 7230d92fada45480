// The shares of ray queries (csrc/query_share.h): every ray of a query has one warp of the
// launch, for grids below, at and above the spread, and for the longest query there can be.
// Prints "ok <queries>" or the first query that leaves rays out.
#include <climits>
#include <cstdio>
#include <initializer_list>

#include "query_share.h"

int main() {
    long queries = 0;
    for (int sms : {1, 2, 76, 148, 152, 160})
        for (int warps : {4, 8, 24, 4 * 152, 6 * 152, 7 * 4 * 152, 8 * 4 * 152})
            for (int k = 1; k < 200000; k += k < 300 ? 1 : k / 37) {
                const int share = ptg::QueryShare(k, sms, warps);
                queries++;
                if (share == 0) continue;
                if (share < 1 || share > ptg::kMostShare || (long long)share * warps < k)
                    return std::printf("%d rays, %d SMs, %d warps: %d each\n", k, sms, warps, share), 1;
            }
    for (int n : {INT_MAX, INT_MAX - 1, INT_MAX - 911, 1 << 30})
        if (ptg::QueryShare(n, 152, 4864) != 0) return std::printf("%d rays are not short\n", n), 1;
    // on 152 SMs with 8 blocks of 4 warps each: 4256 warps take up to 31 rays
    if (ptg::QueryShare(4256, 152, 4864) != 1 || ptg::QueryShare(4257, 152, 4864) != 2 ||
        ptg::QueryShare(31 * 4256, 152, 4864) != 31 || ptg::QueryShare(31 * 4256 + 1, 152, 4864) != 0)
        return std::printf("shares on 152 SMs differ\n"), 1;
    std::printf("ok %ld\n", queries);
    return 0;
}
