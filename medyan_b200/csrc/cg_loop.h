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
// Larger networks run in the graph loop. Microseconds of an iteration, resident and
// graph loop, FP64 with fixed-point sums: 25,200 beads 22 and 54, 100,800 47 and 77,
// 201,600 57 and 73, 235,200 61 and 75, 302,400 70 and 79, 348,600 80-103 and 74-90,
// 420,000 91 and 97 (with atomic sums 84 and 78). Whole calls with 40 energy calls,
// resident and graph: 302,400 5.4-5.7 and 5.5-5.7 ms, 348,600 6.2-6.5 and 6.1.
constexpr int kLoopBeads = 310000;
// Larger ones take blocks of 512 threads. 256 and 512: 25,200 beads 21.7 and 22.7 us,
// 52,500 27.7 and 30.7, 76,440 39.1 and 37.0, 100,800 55 and 47, 201,600 63 and 57.
constexpr int kLoopWideBeads = 75000;

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
// Larger replicas run in the packed batch. 16 replicas over 100 energy calls, resident
// and packed: 10,500 beads each 11.4 and 14.1 ms, 18,900 21.3 and 25.0. The line lies
// below where the two meet: 8 replicas of 25,200 16.3 and 21.8, of 63,000 41 and 76.
constexpr int kLoopBatchBeads = 20000;
cudaError_t launch_cg_loop_batch(const LoopArgs* replicas, const int* order, int n, int* queue, int prec, bool fixed,
                                 bool bounded, cudaStream_t s);

}  // namespace mb
