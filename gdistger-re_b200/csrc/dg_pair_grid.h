// Launch shape of a kernel that trains one or two walks to a warp (dg_sgns_negshare.cu).
// Host code without CUDA types.
#pragma once

#include <algorithm>
#include <cstdint>

namespace dgs {

struct PairGrid {
    int blocks, warps;   // warps of a block
    uint32_t walks;      // walks that a warp trains in turn
};

// most: the shape that fills the GPU.  want: the caller's bound on workers (0: none),
// rounded up to whole blocks as the other trainers' launches round it: below a block's
// warps one block of that many, then a walk to a warp, and two where that is not enough.
inline PairGrid pair_grid(uint32_t want, PairGrid most) {
    if (want == 0) return most;
    if (want < (uint32_t)most.warps) return {1, (int)want, 1};
    const uint64_t full = (uint64_t)most.blocks * most.warps;
    const uint32_t walks = want <= full ? 1 : most.walks;
    const uint64_t per_block = (uint64_t)most.warps * walks;
    return {(int)std::min<uint64_t>(most.blocks, (want + per_block - 1) / per_block), most.warps, walks};
}

}  // namespace dgs
