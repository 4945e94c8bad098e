// cg_loop.h — the resident minimizer loop (cg_loop_kernel.cuh): one kernel that runs a
// whole CGMethod::minimize on a team of thread blocks.
#pragma once

#include <vector>

#include "handle.h"

namespace mb {

// What one team needs of its network; pointers into the handle's buffers.
struct LoopArgs {
    ChainDev ch;
    DeviceFF ff;
    int n3;            // coordinate components
    int vb;            // blocks of the vector passes' summation order (vec_blocks, or 1)
    int fixed;         // deterministic force sums
    double *x, *d, *f0, *f1, *min_e;
    double* lo;        // low parts of the force sums, zero at the launch (floating-point sums in two parts only)
    CGState* st;       // parameters in, final state out
    LambdaSet* lam;    // pending step sizes when the loop hands over
    double* eout;      // [2][MEDYAN_FF_COUNT + 1]: energies before and after
    double* e_last;    // MEDYAN_FF_COUNT + 1: as an energy pass at the final coordinates leaves them; may be null
    double* erow;      // [2][kMaxLambda][4][loop_row_count]
    double* vrow;      // [2][vb, or the 8 warps of a single one][4]: of the sums, of max|d|
    int* words;        // kLoopWords words, zero at the launch
    int* status;       // force status bits
};

// words: two pass flags (a pair needs a quadrature fallback), the loop's
// outcome, the grid barrier's counter.
constexpr int kLoopWords = 4;
// words[2] at the end: the minimization is complete; it stopped in the loop
// and the graph loop takes over from *st; it stopped in the setup, nothing is
// changed but the force buffers; a grid barrier gave up.
constexpr int kLoopDone = 0, kLoopHandOver = 1, kLoopRestart = 2, kLoopLost = 3;

constexpr int kLoopCluster = 16;    // teams of up to this many blocks are thread-block clusters
constexpr int kLoopGrid = 148;      // blocks of the largest team, a cooperative grid (one block per SM)
constexpr int kLoopBeads = 350000;  // larger networks run in the graph loop
constexpr int kLoopWideBeads = 75000;  // larger ones take blocks of 512 threads

// Blocks of a team for this network, 0 when the network is better off in the
// graph loop, or the device has no room for the team.
int loop_team(const ChainDev& ch, const DeviceFF& ff, const LoopRoom& room);
// Energy rows of a pass at one step size, and the doubles that the rows and the
// vector passes' sums take.
int loop_row_count(const ChainDev& ch, const DeviceFF& ff);
size_t loop_erow_doubles(int rows);
__host__ __device__ __forceinline__ size_t loop_vrow_doubles(int vb) { return 2 * (size_t)(vb == 1 ? 8 : vb) * 4; }
// Kernel attributes, once per device (the current one); before the first launch.
// room: what the device holds, unless it is set already.
cudaError_t init_cg_loop(LoopRoom& room);
cudaError_t launch_cg_loop(const LoopArgs& a, int prec, int team, cudaStream_t s);
// its parts on blocks of 512 threads (cg_loop_wide.cu)
cudaError_t init_cg_loop_wide(LoopRoom& room);
cudaError_t launch_cg_loop_wide(const LoopArgs& a, int prec, int team, cudaStream_t s);


// The replicas of a batch (arguments on the device; vb = 1, the order of the
// packed batch's sums), taken in the order given, each by one cluster. bounded:
// a call limit bounds the iterations.
constexpr int kLoopBatchBeads = 20000;  // larger replicas run in the packed batch
cudaError_t launch_cg_loop_batch(const LoopArgs* replicas, const int* order, int n, int* queue, int prec, bool fixed,
                                 bool bounded, cudaStream_t s);

}  // namespace mb
