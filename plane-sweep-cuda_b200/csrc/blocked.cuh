// Geometry of the solvers that run several iterations per launch
// (tvl1_block_kernel, sparse_block_kernel): a CTA holds a region of kBlockW
// columns x (kBlockRows x warps) rows on chip; lane l has columns 2l and 2l + 1
// of its warp's kBlockRows rows.  An iteration reads one cell further on every
// side, so of the region only the cells at least `halo` (>= the launch's
// iterations) from its rim are stored, and neighbouring regions overlap by
// twice that.  The halo is even, so that column 0 of the image is always the
// first of a lane's pair.
#pragma once

#include "common.cuh"

namespace mvs {

constexpr int kBlockW = 64, kBlockRows = 2;

struct BlockPlan {
    int iters, warps;   // iterations per launch (even), warps per CTA
};

inline int block_halo(int iters) { return (iters + 1) & ~1; }

inline dim3 block_grid(int w, int h, int iters, int warps)
{
    const int k = block_halo(iters);
    return dim3(ceil_div(w, kBlockW - 2 * k), ceil_div(h, kBlockRows * warps - 2 * k));
}

// More iterations or more warps mean fewer launches or less halo, but also
// more cells on the busiest SM.  A launch takes about `launch_us` plus
// `warp_us` for every iteration and warp on the busiest SM, its loads counting
// as `load_iters` iterations (all measured, see the callers); the pair with the
// smallest such sum for the run is taken, and that sum returned in `us`.
inline BlockPlan block_plan(int w, int h, int niters, int max_warps, double launch_us, double warp_us,
                            int load_iters = 0, double *us = nullptr)
{
    BlockPlan best{2, max_warps};
    double cost = 1e30;
    for (int k = 2; k <= 10; k += 2)
        for (int warps = k + 2; warps <= max_warps; ++warps) {
            const dim3 g = block_grid(w, h, k, warps);
            if (g.y > 65535u) continue;
            const double tiles = ceil((double)g.x * g.y / kSMs);
            const double c = ceil_div(niters, k) * (launch_us + warp_us * (k + load_iters) * warps * tiles);
            if (c < cost) {
                cost = c;
                best = BlockPlan{k, warps};
            }
        }
    if (us) *us = cost;
    return best;
}

}  // namespace mvs
