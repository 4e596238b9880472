// Blocks of the extension kernels of one pass (ga_extend_batch*), from what fits an SM, the launch
// shape and what there is to do.
#pragma once
#include <algorithm>
#include <cstdint>
#include "../../include/graphaligner_gb300.h"

namespace gadev
{

// What of a kernel's blocks of `warps` warps is resident on an SM: `fit` of them have the registers
// and shared memory; the shape's cap counts blocks of warps_per_block warps.
inline uint64_t resident_blocks(const ga_launch_shape& sh, uint64_t fit, uint64_t warps)
{
    if (sh.blocks_per_sm == 0) return fit;
    return std::min<uint64_t>(fit, (uint64_t)sh.blocks_per_sm * sh.warps_per_block / warps);
}

struct LaunchGrid
{
    uint64_t fill;       // blocks of fillWarps warps
    uint64_t medium;     // the second fill's, of one warp: 0 where it does not run
    uint64_t trace;      // of warps_per_block warps
};

// fillFit, mediumFit, traceFit: blocks of each kernel that fit an SM (mediumFit 0: no second fill);
// pending: extensions to run; resumeCap: the most that the first fill hands on to the second.
inline LaunchGrid launch_grid(const ga_launch_shape& sh, uint64_t sms, uint64_t fillFit, uint64_t fillWarps, uint64_t mediumFit, uint64_t traceFit,
    uint64_t pending, uint64_t resumeCap)
{
    const uint64_t wpb = sh.warps_per_block;
    LaunchGrid g;
    g.fill = std::min(sms * resident_blocks(sh, fillFit, fillWarps), std::max<uint64_t>(1, (pending + fillWarps - 1) / fillWarps));
    g.medium = std::min(sms * resident_blocks(sh, mediumFit, 1), resumeCap);
    g.trace = std::min(sms * resident_blocks(sh, traceFit, wpb), std::max<uint64_t>(1, (pending + wpb - 1) / wpb));
    return g;
}

}
