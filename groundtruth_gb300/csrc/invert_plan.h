// The steps of the large fronts' selective inversion (factor.cu).  Host code without CUDA, so that the launches' extents can be
// checked where there is no GPU.
#pragma once
#include <stdint.h>
#include <algorithm>
#include <vector>

namespace gt {

// A step takes `block` own columns of every front that has as many left, and its grids are as wide as the widest of them
// needs.  So the fronts stand in the order of their own columns, and a step's are the first of them: with all fronts in every
// grid the blocks without work outnumbered the others 23 to 1 on the 256 x 256 pair, 320 to 1 on a board whose top front has
// 3391 rows and 5000 to 1 on six planes of 1024 x 1024; now 1.6, 2.7 and 3.8 blocks are launched for each that works.
struct InvertPlan {
    std::vector<int64_t> fronts;       // by their own columns, most first
    std::vector<int> count, max_nf;    // per step: the fronts it has, the rows of the largest
};

inline InvertPlan make_invert_plan(std::vector<int64_t> fronts, const int64_t* nown, const int64_t* nbnd, int block) {
    std::stable_sort(fronts.begin(), fronts.end(), [&](int64_t a, int64_t b) { return nown[a] > nown[b]; });
    InvertPlan P;
    const int64_t most = fronts.empty() ? 0 : nown[fronts[0]];
    P.count.assign((most + block - 1) / block, 0);
    P.max_nf.assign(P.count.size(), 0);
    for (int64_t f : fronts)
        for (int64_t s = 0; s * block < nown[f]; ++s) {
            ++P.count[s];
            P.max_nf[s] = std::max(P.max_nf[s], (int)(nown[f] + nbnd[f]));
        }
    P.fronts = std::move(fronts);
    return P;
}

}  // namespace gt
