// Which block of k64_moments_poisson does what.
//
// Blocks are handed out in index order as SMs come free, and one that waits keeps its SM.  So
// nothing that waits may come before something it waits for: the first block forms columns
// (by tickets, all of them if no other gets an SM), the summing blocks follow, which need
// column blocks alone, then the solves, which need summing blocks, then the other column
// blocks, on every SM that is left.  With the solves and up to 24 summing blocks first, a GPU
// of so few SMs (a partition, or one that other processes' launches hold) would have been
// full of waiting blocks.
#pragma once
#include "vx_common.hpp"

namespace vx {

enum PipeRole : int { kPipeColumns = 0, kPipeSummer = 1, kPipeSolver = 2 };
struct PipeBlock {
    PipeRole role;
    int run;  // kPipeSolver: the run it solves
};

VX_HD inline PipeBlock pipe_block(int block, int nruns, int summers) {
    const int b = block - 1;
    if (b < 0 || b >= summers + nruns) return {kPipeColumns, -1};
    if (b < summers) return {kPipeSummer, -1};
    return {kPipeSolver, b - summers};
}

}  // namespace vx
