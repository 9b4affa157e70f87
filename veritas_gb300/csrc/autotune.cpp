// Tile-shape autotuner for the FCT sub-step kernels.
//
// Every FCT kernel walks a list of tiles, one thread block per tile of tile_j (p, the
// coalesced axis) x tile_i (x) cells.  The best shape depends on the patch sizes of the
// set (ragged edges, occupancy, register pressure of the precision's kernels), so the
// engine measures it: for each candidate the tile list is rebuilt and the kernels of a
// step's first FCT stage, as the set's step launches them, are timed with CUDA events on
// the engine's stream; the fastest shape is kept for the set and becomes the default for new
// sets of the same precision.  Their outputs are recomputed before being read in the next
// step, but for the update's f1, which is led to a plane of the limiter's coefficients
// instead (each of them is written before it is read).  The tile shape changes no arithmetic.
#include <array>

#include "engine.hpp"

namespace vx {

std::pair<int, int> Engine::autotune(const std::vector<Run *> &set, int reps) {
    static const int kShapes64[][2] = {{32, 4}, {32, 8}, {32, 16}, {64, 4}, {64, 8}, {128, 2}, {128, 4}};
    // FP32: 128 p cells (four per thread) by 1 .. 16 rows
    static const int kShapes32[][2] = {{128, 1}, {128, 2}, {128, 4}, {128, 8}, {128, 16}};
    LaunchSet &L = get_set(set);
    FctLaunch fl{};
    fl.patches = L.dpatch.p;
    fl.fields = L.dfields.as<RunFields>();
    fl.params = L.dparams.as<double>();
    fl.params32 = L.dparams32.as<float>();
    fl.step = 0;
    fl.stream = stream;
    std::vector<PatchT<double>> spare = L.hpatch;
    for (auto &d : spare) d.f1 = d.Cx;
    DevBuf dspare = upload(spare, stream);
    FctLaunch up = fl;
    up.patches = dspare.p;
    int launched = 0;
    auto sub = [&](const FctLaunch &f, int which, int part = 0) {
        FctLaunch g = f;
        g.part = part;
        if (L.precision == kF32) launch_fct32_substep(g, which);
        else if (L.fast64) launch_fct64_substep_fast(g, which);
        else launch_fct64_substep(g, which);
        launched++;
    };
    auto run_subs = [&]() {
        if (L.precision == kF32) {
            for (int which : {kSubXFlux, kSubPFlux, kSubDS}) sub(fl, which);
        } else {
            sub(fl, kSubGamma);
            sub(fl, kSubFaces, 1);
            sub(fl, kSubFlux, 1);
            const bool lu = L.poisson == kPoissonLU;  // the p faces in two halves around the solve
            sub(fl, kSubFaces, lu ? 4 : 2);
            sub(fl, kSubFlux, lu ? 8 : 2);
        }
        sub(fl, kSubF2);
        sub(fl, kSubLimR);
        sub(up, kSubCUpdate);
    };
    double best_ms = 1e300;
    int best[2] = {L.tile_j, L.tile_i};
    std::vector<std::array<int, 2>> shapes;
    if (L.precision == kF32)
        for (auto &sh : kShapes32) shapes.push_back({sh[0], sh[1]});
    else
        for (auto &sh : kShapes64) shapes.push_back({sh[0], sh[1]});
    for (auto &sh : shapes) {
        L.tile_j = sh[0];
        L.tile_i = sh[1];
        build_tiles(L);  // reallocates every tile list: take the pointers afresh
        fl.tiles = L.dtiles.as<TileRef>();
        fl.ntiles = L.ntiles;
        fl.xtiles = L.dxtiles.as<TileRef>();
        fl.ptiles = L.dptiles.as<TileRef>();
        fl.nxtiles = L.nxtiles;
        fl.nptiles = L.nptiles;
        fl.strip_rows = L.strip_rows;
        fl.tile_j = L.tile_j;
        fl.tile_i = L.tile_i;
        up = fl;
        up.patches = dspare.p;
        run_subs();  // warm-up
        if (cudaGetLastError() != cudaSuccess) continue;  // shape not launchable here
        timer_begin();
        for (int r = 0; r < reps; r++) run_subs();
        const double ms = timer_end() / reps;
        if (ms < best_ms) {
            best_ms = ms;
            best[0] = sh[0];
            best[1] = sh[1];
        }
    }
    L.tile_j = best[0];
    L.tile_i = best[1];
    build_tiles(L);
    if (L.graph) {  // the captured step holds the old tile list
        cudaGraphExecDestroy(L.graph);
        L.graph = nullptr;
    }
    kernel_launches += launched;
    tile_pref[L.precision == kF32][0] = best[0];
    tile_pref[L.precision == kF32][1] = best[1];
    sync();
    return {best[0], best[1]};
}

}  // namespace vx
