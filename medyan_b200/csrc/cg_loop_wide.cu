// cg_loop_wide.cu — the resident minimizer loop on blocks of 512 threads: the
// larger single networks, and the replicas of a batch.
#define LOOP_THREADS 512
#include "cg_loop_kernel.cuh"

namespace mb {

cudaError_t init_cg_loop_wide(LoopRoom& room) { return init_kernels<true>(room); }

cudaError_t launch_cg_loop_wide(const LoopArgs& a, int prec, int team, cudaStream_t s) {
    return launch_single(a, prec, team, s);
}

// Blocks per replica: as many as let every replica have its cluster at once,
// and at least two. A block's instructions per second fall as clusters grow
// (128 replicas of 200-4000 cylinders over 50 iterations: 12.3, 7.8, 9.7, 14.3
// ms with 1, 2, 4, 8 blocks), but a batch that runs to its tolerances ends with
// its longest minimization, alone on its cluster, so those take at least four
// (256 replicas: 743, 491, 361, 371 ms).
static int batch_team(int n, bool bounded) {
    int team = bounded ? 2 : 4;
    while (team < kLoopCluster && 2 * team * n <= kLoopGrid) team *= 2;
    return team;
}

cudaError_t launch_cg_loop_batch(const LoopArgs* replicas, const int* order, int n, int* queue, int prec, bool fixed,
                                 bool bounded, cudaStream_t s) {
    const int team = batch_team(n, bounded);
    if (prec == MEDYAN_PREC_MIXED)
        return fixed ? launch_batch<float, true>(replicas, order, n, queue, team, s)
                     : launch_batch<float, false>(replicas, order, n, queue, team, s);
    return fixed ? launch_batch<double, true>(replicas, order, n, queue, team, s)
                 : launch_batch<double, false>(replicas, order, n, queue, team, s);
}

}  // namespace mb
