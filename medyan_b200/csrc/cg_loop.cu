// cg_loop.cu — the resident minimizer loop on blocks of 256 threads, and the
// rules that choose where a minimization runs.
#define LOOP_THREADS 256
#include "cg_loop_kernel.cuh"

#include <mutex>

namespace mb {

// Which networks run here, and on how many blocks: one for every eight force
// tasks and every energy round of a pass with one step size, so that a small
// network's work all runs at once, up to one block per SM.
//
// A cluster's barrier takes 0.7 us where the grid's takes 1.2, so teams of up
// to 16 blocks (the largest cluster) are clusters. The graph loop takes over
// where its kernels, which hold three to four times as many threads per SM,
// are faster, and where the device does not hold the team at once (fewer SMs): a
// launch would be refused.
int loop_team(const ChainDev& ch, const DeviceFF& ff, const LoopRoom& room) {
    if (ch.n_pos <= 0 || ch.n_pos > kLoopBeads) return 0;
    auto chunks = [](int n, int per) { return (n + per - 1) / per; };
    const int tasks = chunks(ff.n_excl, 8) + chunks(ff.n_branch, 32) + chunks(ff.n_stretch, 32) + chunks(ff.n_bend, 32) +
                      chunks(ff.n_linker, 32) + chunks(ff.n_motor, 32) + chunks(ff.n_boundary, 32) +
                      chunks(ch.n_pos, kWarpOut);
    const int rows = loop_row_count(ch, ff);
    if (rows > kMaxRows) return 0;
    const int blocks = chunks(tasks, kWarps) + rows;
    int team = 1;
    while (team < blocks && team < kLoopCluster) team *= 2;
    if (blocks > kLoopCluster) team = blocks < kLoopGrid ? blocks : kLoopGrid;
    return team <= (blocks > kLoopCluster ? room.grid : room.cluster) ? team : 0;
}

int loop_row_count(const ChainDev& ch, const DeviceFF& ff) {
    int n = 0;
    for (int kind = 0; kind < kEKinds; ++kind) n += loop_rows(ch, ff, kind);
    return n;
}

size_t loop_erow_doubles(int rows) { return 2 * (size_t)kMaxLambda * kRowVals * rows; }

cudaError_t init_cg_loop(LoopRoom& room) {
    static std::mutex mu;
    static LoopRoom rooms[64];
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(mu);
    if (rooms[dev].grid < 0) {
        LoopRoom r;
        r.cluster = kLoopCluster;
        r.grid = kLoopGrid;
        e = init_kernels<false>(r);
        if (e == cudaSuccess) e = init_cg_loop_wide(r);
        if (e != cudaSuccess) return e;
        rooms[dev] = r;
    }
    if (room.grid < 0) room = rooms[dev];
    return cudaSuccess;
}

cudaError_t launch_cg_loop(const LoopArgs& a, int prec, int team, cudaStream_t s) {
    return a.n3 > 3 * kLoopWideBeads ? launch_cg_loop_wide(a, prec, team, s) : launch_single(a, prec, team, s);
}

}  // namespace mb
