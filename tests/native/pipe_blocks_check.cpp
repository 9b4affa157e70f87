// Runs the block order of the pipelined moments + solve launch (pipe_blocks.hpp) on S SMs, a
// block each, blocks handed out in index order as SMs come free, for every S from 1 to more
// than the grid.  A column block always ends; a summing block once a column block has run or
// runs; a solve once a summing block has run or runs.  Fails where blocks that cannot end
// hold every SM, or where the grid lacks a run's solve or a summing block.
#include <cstdio>
#include <vector>

#include "pipe_blocks.hpp"

int main() {
    int checked = 0;
    for (int nruns = 1; nruns <= 4; nruns++)
        for (int summers = 1; summers <= 24; summers++)
            for (int workers : {1, 2, 7, 150}) {
                const int grid = nruns + summers + workers;
                std::vector<int> solves(nruns, 0);
                int ns = 0, nc = 0;
                for (int b = 0; b < grid; b++) {
                    const vx::PipeBlock me = vx::pipe_block(b, nruns, summers);
                    if (me.role == vx::kPipeSolver) {
                        if (me.run < 0 || me.run >= nruns || solves[me.run]++) return std::printf("bad run\n"), 1;
                    } else {
                        (me.role == vx::kPipeSummer ? ns : nc)++;
                    }
                }
                for (int s : solves)
                    if (s != 1) return std::printf("run without a solve\n"), 1;
                if (ns != summers || nc != workers) return std::printf("wrong counts\n"), 1;
                for (int sms = 1; sms <= grid + 1; sms++, checked++) {
                    std::vector<int> on;
                    int next = 0, seen[3] = {0, 0, 0};
                    while (next < grid || !on.empty()) {
                        while (next < grid && (int)on.size() < sms) {
                            on.push_back(vx::pipe_block(next++, nruns, summers).role);
                            seen[on.back()]++;
                        }
                        std::vector<int> left;
                        for (int role : on) {
                            const bool ends = role == vx::kPipeColumns || (role == vx::kPipeSummer && seen[vx::kPipeColumns]) ||
                                              (role == vx::kPipeSolver && seen[vx::kPipeSummer] && seen[vx::kPipeColumns]);
                            if (!ends) left.push_back(role);
                        }
                        if (left.size() == on.size()) {
                            std::printf("%d runs, %d summing, %d column blocks: %d SMs full of waiting blocks\n", nruns, summers,
                                        workers, sms);
                            return 1;
                        }
                        on.swap(left);
                    }
                }
            }
    std::printf("%d grids end\n", checked);
    return 0;
}
