// pbatch.h — the packed layout of a batch of independent networks.
//
// All replicas' beads, chains and interaction records are concatenated into
// one set of device arrays, so every force and energy kernel runs once per
// pass for the whole batch. Each replica's records of a force field are
// padded to whole blocks (padding records carry bead offset -1 and are
// skipped), so every block of the energy kernels belongs to one replica and
// its partial sums are that replica's. The conjugate-gradient state, the
// line-search step sizes and the reductions of the vector passes are per
// replica (cg.cu, batched kernels).
#pragma once

#include <vector>

#include "cg_loop.h"
#include "handle.h"

namespace mb {

struct PackedBatch {
    int R = 0;                        // replicas
    int nb = 0;                       // packed beads
    std::vector<int> base;            // bead base of each replica (R + 1)
    DevBuf<int> base_dev;             // the same on the device
    long long gen = -1;               // sum of the replicas' ff_gen at packing

    // records (internal bead order of each replica, offsets shifted by 3 * base)
    DevBuf<unsigned char> flags;
    DevBuf<double2> link_p, bend_p;
    DevBuf<int2> stretch_bs;
    DevBuf<double2> stretch_p;
    DevBuf<int4> bend_bs;
    DevBuf<double2> bend_pp;
    DevBuf<int4> linker_bs, motor_bs, branch_bs, excl_bs;
    DevBuf<double4> linker_p, motor_p, branch_pa, branch_pb, planes;
    DevBuf<double> excl_krs;
    DevBuf<int> boundary_bs, boundary_plane;
    DevBuf<double2> boundary_p;
    DeviceFF ff{};
    ChainDev ch{};
    // launch shapes of the packed layout (medyan_batch_set_shapes): records
    // per bonded block and pairs per excluded-volume block (each replica's
    // records are padded to whole blocks), chain force threads per block,
    // positions per chain energy block
    int bonded_block = kBlock, excl_block = kExclBlock, chain_threads = 256, chain_chunk = 256;
    bool repack = false;  // shapes changed since the last packing

    // per-replica block and row tables
    DevBuf<int4> chain_table;         // chain energy block -> (replica, first, end position)
    int n_chain_blocks = 0;
    DevBuf<int> rows;                 // chain[R+1] | seg[6][R+1] | excl[R+1] | excl pairs[R+1]
    DevBuf<int> rep_bead, rep_bonded, rep_excl;  // replica of each position / bonded block / excl block
    DevBuf<int> act;                  // replicas taking part in the current pass

    // energy / force scratch
    EnergyScratch es{};
    ForceScratch fs{};
    DevBuf<double> partial;
    DevBuf<int> e_fb_count, e_bad, f_fb_count, f_fb_list, force_status;
    DevBuf<int2> e_fb_list;

    // conjugate gradient
    DevBuf<double> x, d, dS, fcur, fnew, minE, out, eout, one;
    DevBuf<CGState> st;
    DevBuf<LambdaSet> Lr, Lg, Lzero;
    DevBuf<double> lam0;
    DevBuf<int> off;
    cudaGraphExec_t graph = nullptr;
    int graph_prec = -1;
    long long graph_gen = -1;
    // fixed-point force sums (medyan_batch_set_deterministic); the graph
    // is rebuilt when it changes
    bool deterministic = false;
    bool graph_det = false;

    // resident loop (cg_loop_kernel.cuh): a replica per cluster, on its handle's own
    // records and these vectors; arguments, control words, sums' rows, the
    // order of the queue, pinned staging of coordinates and forces
    DevBuf<LoopArgs> loop_args;
    DevBuf<int> loop_words, loop_order;
    DevBuf<double> loop_rows, lx, ld, lf0, lf1, lmin, llo, leout;
    DevBuf<CGState> lst;
    DevBuf<LambdaSet> llam;
    std::vector<int> lbase;           // bead base of each replica (R + 1)
    long long loop_gen = -1;          // the replicas' generations and settings of loop_args
    bool loop_fixed = false;
    unsigned char* pinned = nullptr;
    size_t pinned_bytes = 0;

    cudaStream_t stream = nullptr;
    Fork fork{};

    const int* rows_chain() const { return rows.raw(); }
    const int* rows_seg() const { return rows.raw() + (R + 1); }
    const int* rows_excl() const { return rows.raw() + 7 * (R + 1); }
    const int* excl_pairs() const { return rows.raw() + 8 * (R + 1); }

    ~PackedBatch();
};

// Builds (or rebuilds) the packed arrays from the replicas' handles.
medyan_status pack_batch(PackedBatch& pb, const std::vector<medyan_mech*>& h);
// The stream and side streams, made once.
medyan_status batch_streams(PackedBatch& pb);
// Whether the resident loop takes this batch (cg_loop_kernel.cuh), and one batched
// minimization there: coordinates in and out of the callers' arrays, the state
// and energies of replica r into st[r] and eout + 2 r (MEDYAN_FF_COUNT + 1).
// outcome[r] is not kLoopDone for a replica that met a pair which needs a
// quadrature: nothing of it is written but, at kLoopHandOver, the state that the
// packed run goes on from.
bool batch_loop_takes(const std::vector<medyan_mech*>& h);
medyan_status batch_loop_run(PackedBatch& pb, const std::vector<medyan_mech*>& h, const medyan_cg_params* p,
                             double* const* coords, double* const* forces, CGState* st, double* eout, int* outcome,
                             int* force_status);
// The start state of a replica with nb beads.
CGState batch_start_state(const medyan_cg_params* p, int nb);
// A minimization in progress (the resident loop's) that a packed run goes on with.
struct PackedCarry {
    int r;                            // its replica in the packing
    CGState st;
    const double *x, *d, *f, *min_e;  // on the device, the replica's beads
    const LambdaSet* lam;             // step sizes of the pending pass
    const double* eout;
};
// Its replica r of pb's last resident run, for replica `to` of a packing.
PackedCarry batch_loop_carry(const PackedBatch& pb, int r, const CGState& st, int to);
// Runs one batched minimization on the packed arrays (coordinates already in
// pb.x), of the replicas in carry from where they stand; results stay on the
// device (pb.x, pb.fcur, pb.st, pb.eout).
medyan_status cg_batch_run(PackedBatch& pb, int prec, const medyan_cg_params* p,
                           const std::vector<PackedCarry>& carry = {});
// Mean time (ms) of one packed evaluate (energy and forces of every replica
// at pb.x) after two warm-up passes; for the autotuner.
medyan_status cg_batch_time_evaluate(PackedBatch& pb, int prec, int reps, float* ms);

}  // namespace mb
