// cg_loop_kernel.cuh — CGMethod::minimize (src/Mechanics/Minimizer/CGMethod.hpp:826-1743)
// as one resident kernel.
//
// A team of blocks (a thread-block cluster, or a cooperative grid) keeps
// running from the first energy to the last: every step of an iteration is a
// phase of the kernel, and a team barrier stands where the graph loop (cg.cu)
// has kernel boundaries. An iteration whose line search takes the predicted
// trial has two:
//
//   pass   energies at the trial step sizes, and the forces at the trial the
//          previous line search took, side by side                  | barrier
//   dots   every block adds the energy rows and decides; then, per component,
//          d = F + beta d, x += lambda d, and the sums F'.F', F'.F, d.F',
//          max|F'| of the new force F'                              | barrier
//
// and the next pass begins with every block adding the rows of the sums. The
// direction F' + beta d is not stored before the next dots phase: a pass forms
// it where it gathers a bead (x, F' and d instead of x and d), which saves the
// direction's own phase. Its slope d.F is F'.F' + beta d.F'; the slope only
// enters comparisons.
//
// No block waits for another's decision: thread 0 of each block runs the same
// scalar code (cg_scalar.cuh) on the same sums, on the block's own copy of the
// state in shared memory, so a barrier is all the blocks exchange.
//
// The path is the graph loop's bit for bit with deterministic force sums: the
// potentials are the same expressions, the vector sums that beta is made of
// keep the order of the vector passes (vec_blocks), and energies are added in
// the order of the energy kernels and their finish (a deep line search compares
// energies that differ by their last bits). Only the slope is summed otherwise,
// and it only enters comparisons with differences of energies.
//
// Included with LOOP_THREADS, the threads of a block, by one file per size
// (cg_loop.cu, cg_loop_wide.cu): 256 threads have up to 255 registers each and
// the shorter tasks, 512 have 128 and hide more latency once every warp has
// several tasks.
//
// What it leaves to the graph loop: a pair that the analytic excluded-volume
// formulas reject. Its quadrature is long and rare, so the loop stops in front
// of the pass and hands its state over.
#include <cooperative_groups.h>

#include "cg_loop.h"
#include "cg_scalar.cuh"
#include "excl_quad.cuh"
#include "records.cuh"

namespace mb {
namespace {

constexpr int kLoopThreads = LOOP_THREADS;
constexpr int kWarps = kLoopThreads / 32;
constexpr int kSlots = MEDYAN_FF_COUNT;
constexpr int kRowVals = 4;                             // energies of a row: a branch row's four potentials
constexpr int kFinishShares = kFinishBlocks;            // shares of the rows that the energy finish adds apart
constexpr int kMaxRows = kFinishShares * 256;           // rows that a share adds in one round
constexpr int kVecGroups = kLoopThreads / kVecThreads;  // virtual blocks a block works on at once
constexpr int kVecSlots = 8;                            // and between two barriers of the block
// Polls before a grid barrier gives up (a poll is one L2 round trip, so this
// is tens of seconds; blocks are resident together and arrive in microseconds).
constexpr int kBarrierPolls = 1 << 25;

// Kinds of work in a pass. Rows are in the energy kernels' order: chain,
// leftover stretches and bends, linkers, motors, branch points, boundary terms,
// cylinder pairs.
enum { FX, FB, FC, FLinker, FMotor, FBoundary, FStretch, FBend, kFKinds };
enum { EX, EC, EB, ELinker, EMotor, EBoundary, EStretch, EBend, kEKinds };

// The kind of each slot's rows (filament slots: the leftovers), four bits apiece.
constexpr unsigned long long kSlotKind =
    (unsigned long long)EStretch << (4 * MEDYAN_FF_FILAMENT_STRETCHING) |
    (unsigned long long)EBend << (4 * MEDYAN_FF_FILAMENT_BENDING) |
    (unsigned long long)ELinker << (4 * MEDYAN_FF_LINKER_STRETCHING) |
    (unsigned long long)EMotor << (4 * MEDYAN_FF_MOTOR_STRETCHING) |
    (unsigned long long)EB << (4 * MEDYAN_FF_BRANCHING_STRETCHING) |
    (unsigned long long)EB << (4 * MEDYAN_FF_BRANCHING_BENDING) |
    (unsigned long long)EB << (4 * MEDYAN_FF_BRANCHING_DIHEDRAL) |
    (unsigned long long)EB << (4 * MEDYAN_FF_BRANCHING_POSITION) |
    (unsigned long long)EX << (4 * MEDYAN_FF_EXCLUDED_VOLUME) | (unsigned long long)EBoundary << (4 * MEDYAN_FF_BOUNDARY);

// Rows (blocks of the energy kernels) of one kind.
__host__ __device__ inline int loop_rows(const ChainDev& ch, const DeviceFF& ff, int kind) {
    const int n = kind == EX ? ff.n_excl : kind == EC ? ch.n_pos : kind == EB ? ff.n_branch : kind == ELinker ? ff.n_linker
                : kind == EMotor ? ff.n_motor : kind == EBoundary ? ff.n_boundary : kind == EStretch ? ff.n_stretch : ff.n_bend;
    const int per = kind == EX ? kExclBlock : kBlock, b = (n + per - 1) / per;
    return kind == EC && b > 148 * 4 ? 148 * 4 : b;  // the chain kernel's grid is capped (chain_blocks)
}
static_assert(kBlock == kVecThreads && kExclBlock == 64, "the rounds of a pass make the energy kernels' rows");

struct Team {
    int rank, size;
    bool cluster;
    unsigned* bar;
    unsigned target;  // thread 0: arrivals that end the current grid barrier
};

// A block's shared memory. The arguments are here too: a team barrier drops
// what the L1 cache holds, so fields read through a reference to the kernel's
// parameters would come from the L2 cache after every one.
struct Smem {
    LoopArgs a;
    Team tm;
    CGState s;
    LambdaSet L;
    int rows[kEKinds], row0[kEKinds];   // rows of each energy kind, and the first of them
    int n_rows;
    int n_trees;                        // trees of the energy finish that have rows of their slot:
    unsigned short tree[kFinishShares * 8 * kSlots];  // slot, share and 32 rows of the share (16, 8 and 1 apart)
    double esum[2][kWarps][kRowVals];   // warp sums of the energy rounds (a group's rounds alternate)
    double part[kMaxLambda * kSlots][kFinishShares * 8];  // sums over 32 rows each, per step size and slot
    double out[kMaxLambda * kOut];  // energies per step size: slots, then the total
    alignas(16) double red[4 * 8];
    alignas(16) double vred[kVecSlots][8][4];   // warp sums of the virtual blocks in flight
    double beta;      // the direction is F + beta d
    int spec_on;      // the next pass computes the speculative force
    int dirty;        // the next force buffer holds a speculative force
    int hit;          // the speculative force is the one the iteration needs
    int min_pending;  // x is the lowest-energy point and not yet copied to min_e
    int lost;         // a grid barrier gave up
    int job;          // the replica this cluster takes next
};

__device__ __forceinline__ Smem& smem() {
    extern __shared__ __align__(16) unsigned char loop_smem[];
    return *reinterpret_cast<Smem*>(loop_smem);
}

// Team barrier: what any thread of the team wrote before it is visible to all
// after it. False when a grid barrier gave up (the kernel then ends).
__device__ __forceinline__ bool team_sync() {
    Smem& sm = smem();
    Team& t = sm.tm;
    if (t.cluster) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        t.target += t.size;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(t.bar) : "memory");
        unsigned v = 0;
        int polls = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(t.bar) : "memory");
        } while ((int)(v - t.target) < 0 && ++polls < kBarrierPolls);
        if ((int)(v - t.target) < 0) sm.lost = 1;
    }
    __syncthreads();
    return !sm.lost;
}

// Positions x, or x + lam (F + beta d), of arrays that change during the
// kernel: plain loads.
struct Pos {
    const double* x;
    const double* d;
    const double* F;
    double beta, lam;
    bool move;
    __device__ __forceinline__ V3 operator()(int o) const {
        const V3 p{x[o], x[o + 1], x[o + 2]};
        if (!move) return p;
        const V3 g{F[o], F[o + 1], F[o + 2]}, q{d[o], d[o + 1], d[o + 2]};
        return move3(p, lam, V3{g.x + beta * q.x, g.y + beta * q.y, g.z + beta * q.z});
    }
};

// Floating-point sums in two parts: v's multiple of 2^-26 is added to the force, the rest to lo.
// The first sums are exact (below 2^27), whatever the order in which the team's
// blocks add; the second vary by rounding of parts below 2^-27, 1e-24 pN. Added
// as they are, a bead's three or more contributions gave other last bits from run to
// run, and a minimization by chance reaches its tolerance on another path: of 400
// minimizations of 12 filaments of 6 cylinders 31 to 41 ended far from the oracle's
// energy; now none, all alike. It costs 3 to 6 % of a minimization (550 beads 852 and 908
// us, 10,500 897 and 970, 52,500 1,970 and 2,085, a batch of 128 replicas 6.8 and 7.1 ms),
// at 100,800 beads 13 %, and larger networks' sums differ from run to run in every
// form: the 512-thread blocks of a single network add as it is (kParts).
template <bool BATCH>
constexpr bool kParts = BATCH || kLoopThreads == 256;
constexpr double kHiCenter = 1.5 * 67108864.0, kHiRange = 33554432.0;
__device__ __forceinline__ void add_parts(double* f, double* lo, double v) {
    const bool in = fabs(v) < kHiRange;  // else as it is (NaN and infinities too)
    const double h = in ? __dadd_rn(__dadd_rn(v, kHiCenter), -kHiCenter) : v;
    const double l = in ? v - h : 0.0;
    red_add(f, h);
    if (l != 0.0) red_add(lo, l);
}

// Force target with the kind of sums fixed at compile time: half the code of
// every addition, in a kernel that is bound by fetching its instructions.
template <bool FIXED, bool PARTS>
struct Sink {
    int* status;
    double* lo;
};
template <bool FIXED, bool PARTS, class R>
__device__ __forceinline__ void target_add(const Sink<FIXED, PARTS>& t, double* f, int off, R fx, R fy, R fz) {
    if constexpr (FIXED) {
        red_add_fixed(f + off, fixed_of(double(fx), t.status));
        red_add_fixed(f + off + 1, fixed_of(double(fy), t.status));
        red_add_fixed(f + off + 2, fixed_of(double(fz), t.status));
    } else if constexpr (PARTS) {
        add_parts(f + off, t.lo + off, double(fx));
        add_parts(f + off + 1, t.lo + off + 1, double(fy));
        add_parts(f + off + 2, t.lo + off + 2, double(fz));
    } else {
        add_force(f, off, fx, fy, fz);
    }
}

// Chain tile w: lanes hold centres 30w-1 .. 30w+30.
template <class R, bool E, bool F, class Target>
__device__ __forceinline__ void chain_tile(const ChainDev& ch, const Target& t, const Pos& P, double* f, int w,
                                           double& es, double& eb) {
    const int n = ch.n_pos, lane = threadIdx.x & 31;
    const int q = w * kWarpOut - 1 + lane;
    const bool in = q >= 0 && q < n;
    const int qe = lane == 0 ? q - 1 : q + 1;
    V3 c{0.0, 0.0, 0.0}, ce{0.0, 0.0, 0.0};
    if (in) c = P(3 * q);
    if ((lane == 0 || lane == 31) && qe >= 0 && qe < n) ce = P(3 * qe);
    const unsigned fl = in ? __ldg(ch.flags + q) : 0u;
    const double2 lp = in ? __ldg(ch.link_p + q) : double2{0.0, 0.0};
    const double2 bp = in ? __ldg(ch.bend_p + q) : double2{0.0, 0.0};
    V3 cprev = shfl_up3(c), cnext = shfl_down3(c);
    if (lane == 0) cprev = ce;
    if (lane == 31) cnext = ce;
    chain_lane<R, E, F>(cprev, c, cnext, fl, lp, bp, lane >= 1 && lane <= kWarpOut && in, q, t, f, es, eb);
}

// Energies of the link and the bend of position q (32 consecutive positions
// per warp).
__device__ __forceinline__ void chain_energies(const ChainDev& ch, const Pos& P, int q, double& es, double& eb) {
    const int n = ch.n_pos, lane = threadIdx.x & 31;
    const bool in = q < n;
    const int qe = lane == 0 ? q - 1 : q + 1;
    V3 c{0.0, 0.0, 0.0}, ce{0.0, 0.0, 0.0};
    if (in) c = P(3 * q);
    if ((lane == 0 || lane == 31) && qe >= 0 && qe < n) ce = P(3 * qe);
    const unsigned fl = in ? __ldg(ch.flags + q) : 0u;
    const double2 lp = in ? __ldg(ch.link_p + q) : double2{0.0, 0.0};
    const double2 bp = in ? __ldg(ch.bend_p + q) : double2{0.0, 0.0};
    V3 cp = shfl_up3(c), cn = shfl_down3(c);
    if (lane == 0) cp = ce;
    if (lane == 31) cn = ce;
    const T3<double> r = diff<double>(c, cn), r0 = diff<double>(cp, c);
    const double len = sqrt(dot(r, r));
    double before = __shfl_up_sync(kFull, len, 1);
    if (lane == 0) before = sqrt(dot(r0, r0));
    if (fl & kLink) es += stretch_energy_of(len, lp.x, lp.y);
    if (fl & kBend) eb += bend_energy_of<double>(r0, r, before, len, bp.x, bp.y);
}

__device__ __forceinline__ double tree8(const double (*v)[kRowVals], int j) {
    return ((v[0][j] + v[4][j]) + (v[2][j] + v[6][j])) + ((v[1][j] + v[5][j]) + (v[3][j] + v[7][j]));
}

// One pass: energies at the K step sizes of sm.L into the energy rows, and,
// with force, the forces at lam_f added to f. P gives the positions (at x
// itself without a move).
//
// Forces are cut into warp tasks: eight cylinder pairs, 32 records, or a chain
// tile. Energies are cut into rounds, in which eight warps of a block make one
// row: the 256 records, 256 positions or 64 pairs whose energies a block of the
// energy kernels adds, in its order. Tasks and rounds are numbered by kind,
// the long kinds first; consecutive tasks go to the warps of one block, and the
// rounds follow on the blocks after the tasks. An SM so executes few kinds in a
// pass: the kernel's code is several times an SM's instruction cache, and with
// kinds dealt round the blocks a task spent half its time fetching
// instructions (a pass of 2000 filaments of 20 cylinders 13.2 against 11.9 us).
template <class R, bool FIXED, bool PARTS>
__device__ __noinline__ void pass(Pos P, int K, bool force, double lam_f, double* f, int* status, int parity) {
    Smem& sm = smem();
    const LoopArgs& a = sm.a;
    const Team& tm = sm.tm;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quad = lane & 3;
    const DeviceFF& ff = a.ff;
    const Sink<FIXED, PARTS> t{status, a.lo};
    bool bad = false;
    int f_blocks = 0;  // blocks that the force tasks fill
    // The pairs' forces, the longest tasks, take four warps of a block, one per
    // scheduler, where a quarter of the team holds them so: two of their FP64
    // chains on one scheduler wait for each other (11,700 cycles of a pass against
    // 10,500 at 50 filaments of 10 cylinders).
    const bool spread = ((ff.n_excl + 7) / 8 + 3) / 4 * 4 <= tm.size;
    if (force) {
        // lane l: tasks of kind l, and the end of their numbers
        const int n = lane == FX ? ff.n_excl : lane == FB ? ff.n_branch : lane == FC ? a.ch.n_pos : lane == FLinker ? ff.n_linker
                    : lane == FMotor ? ff.n_motor : lane == FBoundary ? ff.n_boundary : lane == FStretch ? ff.n_stretch
                    : lane == FBend ? ff.n_bend : 0;
        const int per = lane == FX ? 8 : lane == FC ? kWarpOut : 32;
        int end = (n + per - 1) / per;
        if (spread && lane == FX) end = (end + 3) / 4 * kWarps;
#pragma unroll
        for (int o = 1; o < kFKinds; o <<= 1) {
            const int v = __shfl_up_sync(kFull, end, o);
            if (lane >= o) end += v;
        }
        const int total = __shfl_sync(kFull, end, kFKinds - 1);
        f_blocks = (total + kWarps - 1) / kWarps;
        P.lam = lam_f;
#pragma unroll 1
        for (int task = tm.rank * kWarps + warp; task < total; task += tm.size * kWarps) {
            const int kind = __popc(__ballot_sync(kFull, end <= task) & ((1u << kFKinds) - 1u));
            const int before = __shfl_sync(kFull, end, kind > 0 ? kind - 1 : 0);
            int i = kind > 0 ? task - before : task;
            double none[4];
            if (kind == FX) {
                if (spread) {
                    if (warp >= 4) continue;
                    i = i / kWarps * 4 + warp;
                }
                const int p = i * 8 + (lane >> 2), pc = min(p, ff.n_excl - 1);
                const int4 q = __ldg(ff.excl_bs + pc);
                const double krs = __ldg(ff.excl_krs + pc);
                // lane j of a pair fetches bead j and gets the force on it
                const int o = quad < 2 ? (quad == 0 ? q.x : q.y) : (quad == 2 ? q.z : q.w);
                const V3 own = P(o);
                T3<double> fo;
                const bool ok = excl_force_quad<sizeof(R) == 8>(quad, quad_lane3(own, 0), quad_lane3(own, 1),
                                                                quad_lane3(own, 2), quad_lane3(own, 3), krs, fo);
                if (p < ff.n_excl) {
                    if (ok) target_add(t, f, o, fo.x, fo.y, fo.z);
                    else bad = true;
                }
            } else if (kind == FB) {
                if (i * 32 + lane < ff.n_branch) branch_record<R, false, true>(ff, t, P, f, i * 32 + lane, none);
            } else if (kind == FC) {
                chain_tile<R, false, true>(a.ch, t, P, f, i, none[0], none[1]);
            } else {
                const int seg = kind < FBoundary ? kind - FLinker + 2 : kind == FBoundary ? 5 : kind - FStretch;
                bonded_record<R, false, true>(ff, t, P, f, seg, i * 32 + lane, none);
            }
        }
    }
    if (K > 0) {
        int rounds = sm.n_rows * K, alt = 0;
        const int group = threadIdx.x / kVecThreads, gthread = threadIdx.x % kVecThreads, gwarp = warp & 7;
        // Up to two rounds a block fit beside the forces, on the blocks without
        // tasks; more go round the whole team. Rounds that come round to the first
        // blocks, which have the pairs, end the pass (12,000 cycles there, 9,600 without;
        // with the spread of the pairs a minimization of 500 x 20 cylinders
        // takes 17.6 ms, before 18.5, of 900 x 13 2.73 and 3.02, of 130 x 15 21.9 and 23.1).
        int first = tm.rank - f_blocks, width = tm.size;
        if (f_blocks < tm.size && rounds <= 2 * kVecGroups * (tm.size - f_blocks)) {
            width -= f_blocks;
            if (first < 0) first = rounds;  // none here
        } else {
            first %= tm.size;
            if (first < 0) first += tm.size;
        }
#pragma unroll 1
        for (int round = first * kVecGroups + group; round < rounds; round += width * kVecGroups, alt ^= 1) {
            int kind = 0, v = round, k = 0;
            while (v >= sm.rows[kind] * K) v -= sm.rows[kind++] * K;
            while (v >= sm.rows[kind]) {
                v -= sm.rows[kind];
                ++k;
            }
            P.lam = sm.L.lam[k];
            double e[kRowVals] = {0.0, 0.0, 0.0, 0.0};
            const int i = v * kVecThreads + gthread;  // record or position of this thread
            if (kind == EX) {
                // 64 pairs: warp 4c + j takes the pairs j, j + 4, ... of 32-pair
                // chunk c, which are those the chunk's sum joins first
                const int p = v * 64 + (gwarp >> 2) * 32 + (gwarp & 3) + (lane & ~3), pc = min(p, ff.n_excl - 1);
                const int4 q = __ldg(ff.excl_bs + pc);
                const double krs = __ldg(ff.excl_krs + pc);
                const V3 own = P(quad < 2 ? (quad == 0 ? q.x : q.y) : (quad == 2 ? q.z : q.w));
                const double U = excl_energy_quad(quad, quad_lane3(own, 0), quad_lane3(own, 1), quad_lane3(own, 2),
                                                  quad_lane3(own, 3), krs);
                if (p < ff.n_excl) {
                    if (excl_energy_bad(U)) bad = true;
                    e[0] = U;
                }
            } else if (kind == EC) {
                for (int q = i; q - lane < a.ch.n_pos; q += sm.rows[EC] * kVecThreads)
                    chain_energies(a.ch, P, q, e[0], e[1]);
            } else if (kind == EB) {
                if (i < ff.n_branch) branch_record<double, true, false>(ff, t, P, f, i, e);
            } else {
                const int seg = kind < EBoundary ? kind - ELinker + 2 : kind == EBoundary ? 5 : kind - EStretch;
                bonded_record<double, true, false>(ff, t, P, f, seg, i, e);
            }
            const int vals = kind == EB ? 4 : kind == EC ? 2 : 1;
#pragma unroll
            for (int j = 0; j < kRowVals; ++j) {
                if (j < vals) {
#pragma unroll
                    for (int o = 16; o > 2; o >>= 1) e[j] += __shfl_down_sync(kFull, e[j], o);
                    if (kind != EX) {
                        e[j] += __shfl_down_sync(kFull, e[j], 2);
                        e[j] += __shfl_down_sync(kFull, e[j], 1);
                    }
                    if (lane == 0) sm.esum[alt][warp][j] = e[j];
                }
            }
            if constexpr (kVecGroups == 1) __syncthreads();
            else asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(kVecThreads) : "memory");
            if (gthread < vals) {
                const double(*w)[kRowVals] = sm.esum[alt] + 8 * group;
                const double sum = kind != EX ? tree8(w, gthread)
                                              : ((w[0][0] + w[2][0]) + (w[1][0] + w[3][0])) +
                                                    ((w[4][0] + w[6][0]) + (w[5][0] + w[7][0]));
                a.erow[((size_t)(parity * kMaxLambda + k) * kRowVals + gthread) * sm.n_rows + sm.row0[kind] + v] = sum;
            }
        }
    }
    if (bad) atomicOr(a.words + parity, 1);
}

// ForceFieldManager::computeEnergy's rule (a force field at or below -1 makes
// the total +inf, ForceFieldManager.cpp:137-176) for the sums in sm.out.
__device__ __forceinline__ void total_energies(int K) {
    Smem& sm = smem();
    if (threadIdx.x < K) {
        double* o = sm.out + threadIdx.x * kOut;
        double tot = 0.0;
        bool inf = false;
#pragma unroll
        for (int s = 0; s < kSlots; ++s) {
            if (o[s] <= -1) inf = true;
            else tot += o[s];
        }
        o[kSlots] = inf ? __longlong_as_double(0x7ff0000000000000ULL) : tot;
    }
    __syncthreads();
}

// After the barrier that follows a pass: whether it met a pair that needs a
// quadrature (the same answer in every block: the flag of this parity is not
// written again before the next barrier), and else the energies: every block
// adds the rows in the order of the energy finish (k_energy_finish: eight
// shares of the rows; in a share, a tree over 32 rows, a tree over eight such
// sums; then the shares in order).
template <bool BATCH>
__device__ __noinline__ bool add_rows(int K, int parity) {
    Smem& sm = smem();
    const LoopArgs& a = sm.a;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int flag = *reinterpret_cast<volatile int*>(a.words + parity);
    if constexpr (BATCH) {
        // a replica of a batch: the batched finish's order (a warp per slot:
        // lanes add every 32nd row of a kind, the chain's after the leftovers',
        // then a tree)
#pragma unroll 1
        for (int c = warp; c < K * kSlots; c += kWarps) {
            const int k = c / kSlots, slot = c % kSlots;
            const int kind = (int)(kSlotKind >> (4 * slot)) & 15, j = kind == EB ? slot - MEDYAN_FF_BRANCHING_STRETCHING : 0;
            auto lane_sum = [&](int kd, int val) {
                const double* row = a.erow + ((size_t)(parity * kMaxLambda + k) * kRowVals + val) * sm.n_rows + sm.row0[kd];
                double v = 0.0;
                for (int r = lane; r < sm.rows[kd]; r += 32) v += row[r];
                return v;
            };
            double v = lane_sum(kind, j);
            if (slot <= MEDYAN_FF_FILAMENT_BENDING) v += lane_sum(EC, slot);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
            if (lane == 0) sm.out[k * kOut + slot] = v;
        }
        if (__syncthreads_or(flag)) return false;
        total_energies(K);
        return true;
    }
    // A tree over 32 rows takes eight lanes, each with the four rows that its two
    // first levels join, and only the trees that have a row of their slot are
    // taken: with a warp per 32 rows and a tree per slot among them, one after
    // another, the sums of 75 rows (500 filaments of 20 cylinders) took 9,200
    // cycles of an iteration's 36,000; now 2,950.
    const int R = sm.n_rows, share = (R + kFinishShares - 1) / kFinishShares, subs = (share + 31) / 32;
    const int trees = sm.n_trees, l8 = lane & 7;
    constexpr int kAhead = 2;  // trees loaded before the first is added
#pragma unroll 1
    for (int base = warp * 4; base < K * trees; base += kAhead * kWarps * 4) {
        double v[kAhead][4];
        int at[kAhead];
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            const int t = base + q * kWarps * 4 + (lane >> 3), tc = min(t, K * trees - 1), k = tc / trees;
            const int id = sm.tree[tc - k * trees], slot = id & 15, b = id >> 7, u = (id >> 4) & 7;
            const int kind = (int)(kSlotKind >> (4 * slot)) & 15, j = kind == EB ? slot - MEDYAN_FF_BRANCHING_STRETCHING : 0;
            const int lo = sm.row0[kind], hi = lo + sm.rows[kind], chain = slot <= MEDYAN_FF_FILAMENT_BENDING ? sm.rows[EC] : 0;
            const int r0 = b * share + u * 32, r1 = min(min(R, (b + 1) * share), r0 + 32);
            const double* row = a.erow + (size_t)(parity * kMaxLambda + k) * kRowVals * R;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = r0 + l8 + 8 * i;
                const int val = r >= lo && r < hi ? j : slot;  // chain rows come first, a value per slot
                v[q][i] = r < r1 && ((r >= lo && r < hi) || r < chain) ? row[(size_t)val * R + r] : 0.0;
            }
            at[q] = t < K * trees ? (k * kSlots + slot) * (kFinishShares * 8) + b * 8 + u : -1;
        }
#pragma unroll
        for (int q = 0; q < kAhead; ++q) {
            double w = (v[q][0] + v[q][2]) + (v[q][1] + v[q][3]);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) w += __shfl_down_sync(kFull, w, o, 8);
            if (l8 == 0 && at[q] >= 0) sm.part[0][at[q]] = w;
        }
    }
    if (__syncthreads_or(flag)) return false;
    // eight lanes per step size and slot: a share each, then the shares in order
#pragma unroll 1
    for (int i0 = warp * 32; i0 < K * kSlots * kFinishShares; i0 += kLoopThreads) {
        const int c = min((i0 + lane) >> 3, K * kSlots - 1), b = lane & 7;
        const double* q = sm.part[c] + 8 * b;
        double w = q[0];
        if (subs > 1) {
            double z[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) z[u] = u < subs ? q[u] : 0.0;
            w = ((z[0] + z[4]) + (z[2] + z[6])) + ((z[1] + z[5]) + (z[3] + z[7]));
        }
        double v = 0.0;
#pragma unroll
        for (int q8 = 0; q8 < kFinishShares; ++q8) v += __shfl_sync(kFull, w, q8, 8);
        if (b == 0) sm.out[c / kSlots * kOut + c % kSlots] = v;
    }
    __syncthreads();
    total_energies(K);
    return true;
}

// Sums and a maximum of a vector pass: F'.F', F'.F, d.F', max|F'|.
struct Sums {
    double a, b, c, m;
};
__device__ __forceinline__ void join(Sums& s, const Sums& o) {
    s.a += o.a;
    s.b += o.b;
    s.c += o.c;
    s.m = dmax_ref(s.m, o.m);
}
// Lane 0 gets the warp's, by the tree of the vector passes.
__device__ __forceinline__ void warp_join(Sums& s) {
#pragma unroll 1
    for (int o = 16; o > 0; o >>= 1) {
        Sums n;
        n.a = __shfl_down_sync(kFull, s.a, o);
        n.b = __shfl_down_sync(kFull, s.b, o);
        n.c = __shfl_down_sync(kFull, s.c, o);
        n.m = __shfl_down_sync(kFull, s.m, o);
        join(s, n);
    }
}
// The same tree over eight warps' sums, by the lanes of a group of eight (all
// 32 lanes call; valid in the group's first lane).
__device__ __forceinline__ void eight_join(Sums& s) {
#pragma unroll 1
    for (int o = 4; o > 0; o >>= 1) {
        Sums n;
        n.a = __shfl_down_sync(kFull, s.a, o, 8);
        n.b = __shfl_down_sync(kFull, s.b, o, 8);
        n.c = __shfl_down_sync(kFull, s.c, o, 8);
        n.m = __shfl_down_sync(kFull, s.m, o, 8);
        join(s, n);
    }
}
__device__ __forceinline__ void put(double* r, const Sums& s) {
    *reinterpret_cast<double2*>(r) = double2{s.a, s.b};
    *reinterpret_cast<double2*>(r + 2) = double2{s.c, s.m};
}
__device__ __forceinline__ Sums get(const double* r) {
    const double2 p = *reinterpret_cast<const double2*>(r), q = *reinterpret_cast<const double2*>(r + 2);
    return Sums{p.x, p.y, q.x, q.y};
}

// One vector pass: load(i) for every component i, then apply(i, loaded, sums).
// A virtual block of 256 threads (vec_blocks) is worked by eight warps of one
// block; with a single virtual block its warps are spread over the team
// instead. Its sums go to a row.
template <class Load, class Apply>
__device__ __forceinline__ void vector_pass(double* rows, Load load, Apply apply) {
    Smem& sm = smem();
    const LoopArgs& a = sm.a;
    const Team& tm = sm.tm;
    constexpr int kAhead = 2;  // components loaded before the first is used
    const int lane = threadIdx.x & 31, stride = a.vb * kVecThreads;
    const bool one = a.vb == 1;
    const int t = threadIdx.x % kVecThreads, g = threadIdx.x / kVecThreads;
    // units: virtual blocks (a group of eight warps each), or warps of the only one
    const int units = one ? 8 : a.vb, per = one ? tm.size * kWarps : tm.size * kVecGroups;
    const int mine = one ? tm.rank * kWarps + (threadIdx.x >> 5) : tm.rank * kVecGroups + g;
    const int most = kVecSlots / kVecGroups;
    for (int u0 = mine - (one ? 0 : g); u0 < units; u0 += per * most) {
#pragma unroll 1
        for (int k = 0; k < most && u0 + k * per + (one ? 0 : g) < units; ++k) {
            const int u = u0 + k * per + (one ? 0 : g);
            Sums s{0.0, 0.0, 0.0, 0.0};
#pragma unroll 1
            for (int i = one ? u * 32 + lane : u * kVecThreads + t; i < a.n3; i += kAhead * stride) {
                decltype(load(0)) v[kAhead];
#pragma unroll
                for (int q = 0; q < kAhead; ++q)
                    if (i + q * stride < a.n3) v[q] = load(i + q * stride);
#pragma unroll
                for (int q = 0; q < kAhead; ++q)
                    if (i + q * stride < a.n3) apply(i + q * stride, v[q], s);
            }
            warp_join(s);
            if (lane == 0) put(one ? rows + 4 * u : sm.vred[k * kVecGroups + g][t >> 5], s);
        }
        if (one) continue;
        __syncthreads();
        if (threadIdx.x < 8 * kVecSlots) {  // eight lanes per virtual block
            const int slot = threadIdx.x >> 3, v = u0 + slot / kVecGroups * per + slot % kVecGroups;
            Sums s = get(sm.vred[slot][threadIdx.x & 7]);
            eight_join(s);
            if ((threadIdx.x & 7) == 0 && v < a.vb) put(rows + 4 * (size_t)v, s);
        }
        if (u0 + per * most < units) __syncthreads();
    }
}

// After the barrier that follows a vector pass: the sums of its rows, in the
// vector passes' order (thread q adds blocks q, q + 256, ..., then a tree).
// Valid in thread 0.
__device__ __noinline__ Sums add_vector_rows(const double* rows) {
    Smem& sm = smem();
    const LoopArgs& a = sm.a;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, vb = a.vb;
    Sums s{0.0, 0.0, 0.0, 0.0};
    if (vb == 1) {
        if (warp == 0) {
            if (lane < 8) s = get(rows + 4 * lane);
            eight_join(s);
        }
        return s;
    }
    if (warp * 32 < vb && warp < 8) {
#pragma unroll 1
        for (int q = threadIdx.x; q < vb; q += kVecThreads) join(s, get(rows + 4 * (size_t)q));
        warp_join(s);
    }
    if (vb > 32) {
        if (lane == 0 && warp < 8) put(sm.red + 4 * warp, s);
        __syncthreads();
        if (warp == 0) {
            s = get(sm.red + 4 * (lane & 7));
            eight_join(s);
        }
    }
    return s;
}

template <class R, bool FIXED, bool BATCH>
__device__ void minimize() {
    Smem& sm = smem();
    const LoopArgs& a = sm.a;
    const Team& tm = sm.tm;
    CGState& s = sm.s;
    constexpr bool PARTS = !FIXED && kParts<BATCH>;
    auto words = [](auto& v) { return reinterpret_cast<int*>(&v); };
    for (int i = threadIdx.x; i < (int)(sizeof(CGState) / 4); i += kLoopThreads) words(s)[i] = words(*a.st)[i];
    if (threadIdx.x == 0) {
        sm.L = LambdaSet{};
        sm.L.K = 1;
        sm.beta = 0.0;
        sm.spec_on = sm.dirty = sm.hit = sm.min_pending = sm.lost = 0;
        int at = 0;
        for (int kind : {EC, EStretch, EBend, ELinker, EMotor, EB, EBoundary, EX}) {
            sm.rows[kind] = loop_rows(a.ch, a.ff, kind);
            sm.row0[kind] = at;
            at += sm.rows[kind];
        }
        sm.n_rows = at;
        sm.n_trees = 0;
    }
    __syncthreads();
    if constexpr (!BATCH) {
        for (int i = threadIdx.x; i < kMaxLambda * kSlots * kFinishShares * 8; i += kLoopThreads) sm.part[0][i] = 0.0;
        const int n = sm.n_rows, share = (n + kFinishShares - 1) / kFinishShares, c = threadIdx.x;
        const int r0 = (c >> 3) * share + (c & 7) * 32, r1 = min(min(n, ((c >> 3) + 1) * share), r0 + 32);
        for (int slot = 0; slot < kSlots && c < kFinishShares * 8; ++slot) {
            const int kind = (int)(kSlotKind >> (4 * slot)) & 15;
            const int lo = sm.row0[kind], hi = lo + sm.rows[kind];
            if (max(r0, lo) < min(r1, hi) || (slot <= MEDYAN_FF_FILAMENT_BENDING && r0 < min(r1, sm.rows[EC])))
                sm.tree[atomicAdd(&sm.n_trees, 1)] = (unsigned short)(c << 4 | slot);
        }
    }
    __syncthreads();
    const int first = tm.rank * kLoopThreads + threadIdx.x, step = tm.size * kLoopThreads;
    int parity = 0;  // of the passes: which energy rows and pass flag the next one uses
    auto current = [&] { return s.parity ? a.f1 : a.f0; };
    auto other = [&] { return s.parity ? a.f0 : a.f1; };
    // Writes the state back (block 0) and ends the kernel with `code`. The
    // graph loop finds the direction and the lowest-energy point in place.
    auto leave = [&](int code) {
        if (code == kLoopHandOver) {
            const double* F = current();
            for (int i = first; i < a.n3; i += step) {
                a.d[i] = F[i] + sm.beta * a.d[i];
                if (sm.min_pending) a.min_e[i] = a.x[i];
            }
        }
        __syncthreads();
        if (tm.rank != 0) return;
        if (threadIdx.x == 0) {
            s.spec_valid = 0;
            s.spec_skip = 1;
            s.force_skip = 0;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < (int)(sizeof(CGState) / 4); i += kLoopThreads) words(*a.st)[i] = words(s)[i];
        if (threadIdx.x == 0) {
            *a.lam = sm.L;
            a.words[2] = code;
        }
    };
    auto record = [&](int which) {
        if (threadIdx.x == 0) {
            double tot = 0.0;
            for (int i = 0; i < kSlots; ++i) tot += sm.out[i];  // computeIndividualEnergies: no -1 rule
            if (tm.rank == 0) {
                for (int i = 0; i < kSlots; ++i) a.eout[which * kOut + i] = sm.out[i];
                a.eout[which * kOut + kSlots] = tot;
            }
            s.num_energy_call++;
            if (which == 0) {
                s.prev_energy = tot;
                s.need_e0 = 1;
            }
        }
    };
    const Pos at_x{a.x, nullptr, nullptr, 0.0, 0.0, false};

    // energies before, and the first force
    pass<R, FIXED, PARTS>(at_x, 1, true, 0.0, other(), a.status, parity);
    if (!team_sync()) return leave(kLoopLost);
    if (!add_rows<BATCH>(1, parity)) return leave(kLoopRestart);
    parity ^= 1;
    record(0);
    __syncthreads();

    for (;;) {
        // dots: the direction, the move, the new force's sums; the buffer of
        // the old force becomes zero for the next one
        const bool moved = !s.done && !s.skip_force;
        if (moved) {
            double *Fn = other(), *Fc = current();
            const double lam = s.lam_move, beta = sm.beta;
            const bool copy = sm.min_pending;
            double *x = a.x, *d = a.d, *min_e = a.min_e, *lo = a.lo;
            struct In {
                double x, d, fn, fc, lo;
            };
            vector_pass(
                a.vrow, [&](int i) { return In{x[i], d[i], Fn[i], Fc[i], PARTS ? lo[i] : 0.0}; },
                [&](int i, In v, Sums& q) {
                    const double dn = v.fc + beta * v.d;  // shiftSearchDir (CGMethod.cpp:356-360)
                    if (copy) min_e[i] = v.x;
                    d[i] = dn;
                    x[i] = move1(v.x, lam, dn);
                    if constexpr (FIXED) {
                        v.fn = double(__double_as_longlong(v.fn)) / kFixedScale;
                        Fn[i] = v.fn;
                    } else if constexpr (PARTS) {
                        v.fn += v.lo;
                        lo[i] = 0.0;
                        Fn[i] = v.fn;
                    }
                    Fc[i] = 0.0;
                    q.a += v.fn * v.fn;
                    q.b += v.fn * v.fc;
                    q.c += dn * v.fn;
                    q.m = dmax_ref(q.m, fabs(v.fn));
                });
            if (tm.rank == 0 && threadIdx.x == 0) a.st->spec_status = 0;
            if (!team_sync()) return leave(kLoopLost);
            const Sums q = add_vector_rows(a.vrow);
            if (threadIdx.x == 0) {
                sm.min_pending = 0;
                dots_tail(s, q.a, q.b, q.m);
                if (s.copy_min_e) sm.min_pending = 1;
                // d.F of the new direction
                s.slope = s.dir_mode ? s.new_grad : s.new_grad + s.beta * q.c;
            }
        } else {
            __syncthreads();
            if (threadIdx.x == 0 && !s.done) s.slope = s.new_grad;  // the line search failed: d = F
        }
        __syncthreads();
        if (s.done) break;
        if (s.safe_mode) {
            // max|d|, which only the recovery step after a second failure needs;
            // its rows are apart: another block may still be adding the sums'. A
            // failed line search leaves its speculative force in the other
            // buffer, which the next pass needs zero
            double* max_rows = a.vrow + loop_vrow_doubles(a.vb) / 2;
            const double* F = current();
            const double beta = s.dir_mode ? 0.0 : s.beta;
            if (!moved)
                for (int i = first; i < a.n3; i += step) {
                    other()[i] = 0.0;
                    if constexpr (PARTS) a.lo[i] = 0.0;
                }
            struct In {
                double f, d;
            };
            vector_pass(
                max_rows, [&](int i) { return In{F[i], a.d[i]}; },
                [&](int, const In& v, Sums& q) { q.m = dmax_ref(q.m, fabs(v.f + beta * v.d)); });
            if (tm.rank == 0 && threadIdx.x == 0) a.st->spec_status = 0;
            if (!team_sync()) return leave(kLoopLost);
            const Sums q = add_vector_rows(max_rows);
            if (threadIdx.x == 0) s.dmax = q.m;
        }
        __syncthreads();  // every thread has read the state that thread 0 now changes
        if (threadIdx.x == 0) {
            sm.beta = s.dir_mode ? 0.0 : s.beta;
            dir_tail(s, sm.L, s.slope, s.dmax);
            if (s.reset_after_dir) sm.beta = 0.0;  // conjugacy lost: d = F
            sm.dirty = sm.hit = sm.spec_on = 0;
            s.spec_valid = 0;
            // the speculative force: at the trial that the previous line
            // search took, when the first pass offers it
            const int j = (s.need_e0 ? 1 : 0) + s.last_backtracks;
            if (!s.done && !s.ls_immediate_fail && j < sm.L.K) {
                s.spec_lam = sm.L.lam[j];
                s.spec_valid = sm.spec_on = sm.dirty = 1;
            }
        }
        __syncthreads();
        if (s.done) break;
        // line search
        const Pos along{a.x, a.d, current(), sm.beta, 0.0, true};
        while (s.ls_active && !s.done) {
            const int K = s.ls_immediate_fail ? 0 : sm.L.K;
            if (K > 0) {
                pass<R, FIXED, PARTS>(along, K, sm.spec_on, s.spec_lam, other(), &a.st->spec_status, parity);
                if (!team_sync()) return leave(kLoopLost);
                if (!add_rows<BATCH>(K, parity)) return leave(kLoopHandOver);
                parity ^= 1;
            } else {
                __syncthreads();
            }
            if (threadIdx.x == 0) {
                ls_decide(s, sm.L, sm.out);
                sm.spec_on = 0;
                if (!s.ls_active) {
                    sm.hit = s.spec_valid && !s.skip_force && s.lam_move == s.spec_lam;
                    if (sm.hit && tm.rank == 0 && a.st->spec_status) *a.status |= a.st->spec_status;
                    s.spec_valid = 0;
                }
            }
            __syncthreads();
        }
        // the force at the accepted step, unless the line search's pass had it
        if (!s.done && !s.skip_force && !sm.hit) {
            double* F = other();
            if (sm.dirty) {
                for (int i = first; i < a.n3; i += step) {
                    F[i] = 0.0;
                    if constexpr (PARTS) a.lo[i] = 0.0;
                }
                if (!team_sync()) return leave(kLoopLost);
            }
            pass<R, FIXED, PARTS>(along, 0, true, s.lam_move, F, a.status, parity);
            if (!team_sync()) return leave(kLoopLost);
            if (!add_rows<BATCH>(0, parity)) return leave(kLoopHandOver);
            parity ^= 1;
        }
    }

    // epilogue: the lowest-energy coordinates after a call limit, the current
    // force into f0, the energies after
    const bool restore =
        s.status != MEDYAN_ERR_LINE_SEARCH && s.call_limit && s.have_min_e && !sm.min_pending;
    const bool copy_f = s.parity != 0;
    for (int i = first; i < a.n3; i += step) {
        if (restore) a.x[i] = a.min_e[i];
        if (copy_f) a.f0[i] = a.f1[i];
    }
    if (threadIdx.x == 0) {
        sm.L.K = 1;
        sm.L.lam[0] = 0.0;
    }
    if (!team_sync()) return leave(kLoopLost);
    // after a failed line search they are not part of the result, but a single
    // network's energy buffer holds those of its coordinates all the same
    const bool failed = s.status == MEDYAN_ERR_LINE_SEARCH;
    if (!failed || a.e_last) {
        pass<R, FIXED, PARTS>(at_x, 1, false, 0.0, nullptr, nullptr, parity);
        if (!team_sync()) return leave(kLoopLost);
        if (!add_rows<BATCH>(1, parity)) return leave(kLoopHandOver);
        if (a.e_last && tm.rank == 0 && threadIdx.x < kOut) a.e_last[threadIdx.x] = sm.out[threadIdx.x];
        if (!failed) record(1);
        __syncthreads();
    }
    leave(kLoopDone);
}

template <class R, bool FIXED, bool CLUSTER>
__global__ void __launch_bounds__(kLoopThreads, 1) k_cg_loop(const __grid_constant__ LoopArgs a) {
    if (threadIdx.x == 0) {
        smem().a = a;
        smem().tm = Team{(int)blockIdx.x, (int)gridDim.x, CLUSTER, reinterpret_cast<unsigned*>(a.words + 3), 0u};
    }
    __syncthreads();
    minimize<R, FIXED, false>();
}

// A batch of independent networks: each cluster minimizes one replica after
// another, taken from a queue in the order given (the largest first), until
// none is left. A replica only ever waits for the blocks of its own cluster.
template <class R, bool FIXED>
__global__ void __launch_bounds__(kLoopThreads, 1)
    k_cg_loop_batch(const LoopArgs* __restrict__ replicas, const int* __restrict__ order, int n, int* __restrict__ queue) {
    namespace cg = cooperative_groups;
    const cg::cluster_group cluster = cg::this_cluster();
    Smem& sm = smem();
    cluster.sync();  // a block's shared memory may be written once the block is known to have started
    for (;;) {
        __syncthreads();
        if (cluster.block_rank() == 0 && threadIdx.x == 0) {
            const int job = atomicAdd(queue, 1);
            for (unsigned b = 0; b < cluster.num_blocks(); ++b) *cluster.map_shared_rank(&sm.job, b) = job;
        }
        cluster.sync();
        const int job = sm.job;
        if (job >= n) break;
        if (threadIdx.x == 0) {
            sm.a = replicas[order[job]];
            sm.tm = Team{(int)cluster.block_rank(), (int)cluster.num_blocks(), true, nullptr, 0u};
        }
        __syncthreads();
        minimize<R, FIXED, true>();
    }
    cluster.sync();  // no block leaves while another may still write its next job
}

template <class R, bool FIXED>
cudaError_t launch_batch(const LoopArgs* replicas, const int* order, int n, int* queue, int team, cudaStream_t s) {
    cudaLaunchConfig_t c{};
    c.blockDim = dim3(kLoopThreads);
    c.dynamicSmemBytes = sizeof(Smem);
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = team;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    c.gridDim = dim3(team);
    int clusters = 0;
    cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, k_cg_loop_batch<R, FIXED>, &c);
    if (e != cudaSuccess) return e;
    if (clusters < 1) return cudaErrorInvalidConfiguration;
    c.gridDim = dim3(team * (n < clusters ? n : clusters));
    return cudaLaunchKernelEx(&c, k_cg_loop_batch<R, FIXED>, replicas, order, n, queue);
}

template <class R, bool FIXED>
cudaError_t launch(const LoopArgs& a, int team, cudaStream_t s) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(team);
    c.blockDim = dim3(kLoopThreads);
    c.dynamicSmemBytes = sizeof(Smem);
    c.stream = s;
    cudaLaunchAttribute at{};
    c.attrs = &at;
    c.numAttrs = 1;
    if (team <= kLoopCluster) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = team;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        return cudaLaunchKernelEx(&c, k_cg_loop<R, FIXED, true>, a);
    }
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    return cudaLaunchKernelEx(&c, k_cg_loop<R, FIXED, false>, a);
}

// A kernel's attributes, and the room for it: the largest cluster, or the blocks
// of a cooperative grid.
template <class Kernel>
cudaError_t init_kernel(Kernel k, bool cluster, LoopRoom& room) {
    if (!cluster) {
        int dev = 0, sms = 0, coop = 0, per = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, kLoopThreads, sizeof(Smem));
        if (e == cudaSuccess && room.grid > (coop ? per * sms : 0)) room.grid = coop ? per * sms : 0;
        return e;
    }
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(kLoopCluster);
    c.blockDim = dim3(kLoopThreads);
    c.dynamicSmemBytes = sizeof(Smem);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kLoopCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &c) != cudaSuccess) {
        cudaGetLastError();  // no such cluster on this device
        n = 0;
    }
    if (n < 1) room.cluster = 0;
    return cudaSuccess;
}

// BATCH: the kernels that take a batch's replicas too.
template <bool BATCH, class R, bool FIXED>
cudaError_t init_kernels_of(LoopRoom& room) {
    cudaError_t e = init_kernel(k_cg_loop<R, FIXED, true>, true, room);
    if (e == cudaSuccess) e = init_kernel(k_cg_loop<R, FIXED, false>, false, room);
    if constexpr (BATCH)
        if (e == cudaSuccess) e = init_kernel(k_cg_loop_batch<R, FIXED>, true, room);
    return e;
}
template <bool BATCH>
cudaError_t init_kernels(LoopRoom& room) {
    cudaError_t e = init_kernels_of<BATCH, float, false>(room);
    if (e == cudaSuccess) e = init_kernels_of<BATCH, float, true>(room);
    if (e == cudaSuccess) e = init_kernels_of<BATCH, double, false>(room);
    if (e == cudaSuccess) e = init_kernels_of<BATCH, double, true>(room);
    return e;
}

cudaError_t launch_single(const LoopArgs& a, int prec, int team, cudaStream_t s) {
    if (prec == MEDYAN_PREC_MIXED) return a.fixed ? launch<float, true>(a, team, s) : launch<float, false>(a, team, s);
    return a.fixed ? launch<double, true>(a, team, s) : launch<double, false>(a, team, s);
}

}  // namespace
}  // namespace mb
