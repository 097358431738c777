// Host-side work division shared by the kernels that give every linear of a launch a contiguous range of CTAs.
#pragma once

namespace nq {

// Deal `grid` CTAs to the jobs of a phase so that the largest per-CTA stream (row groups x chunks) is as small as
// possible: shares in proportion to the work, the rest one by one to the job that is worst off.
inline void deal_ctas(int grid, int n, const int* groups, const int* chunks, int* ncta) {
    long long total = 0;
    for (int i = 0; i < n; ++i) total += (long long)groups[i] * chunks[i];
    int used = 0;
    for (int i = 0; i < n; ++i) {
        long long share = (long long)groups[i] * chunks[i] * grid / total;
        if (share > groups[i]) share = groups[i];
        ncta[i] = share < 1 ? 1 : (int)share;
        used += ncta[i];
    }
    while (used < grid) {
        int best = -1;
        long long best_cost = -1;
        for (int i = 0; i < n; ++i) {
            if (ncta[i] >= groups[i]) continue;      // one row group per CTA already
            const long long cost = (long long)((groups[i] + ncta[i] - 1) / ncta[i]) * chunks[i];
            if (cost > best_cost) { best_cost = cost; best = i; }
        }
        if (best < 0) break;
        ++ncta[best];
        ++used;
    }
    while (used > grid) {      // the minimum of one each may have gone over
        int most = 0;
        for (int i = 1; i < n; ++i) most = ncta[i] > ncta[most] ? i : most;
        --ncta[most];
        --used;
    }
}

}  // namespace nq
