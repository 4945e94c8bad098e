// cg_scalar.cuh — the scalar logic of CGMethod::minimize
// (src/Mechanics/Minimizer/CGMethod.hpp:826-1743) on a CGState: line-search
// decisions, the quadratic line search, beta, direction resets, convergence
// and call limits. One thread runs it, whatever the kernels around it: the
// graph loop's one-thread kernels and last blocks (cg.cu), the packed batch's
// one thread per replica (cg.cu), and thread 0 of every block of the resident
// loop (cg_loop_kernel.cuh), which keeps a copy of the state per block.
#pragma once

#include "handle.h"

namespace mb {
namespace {

constexpr int kVecThreads = 256;         // threads of a vector pass's block
constexpr double kLambdaTol = 1e-8;      // CGMethod::LAMBDATOL (double build)
constexpr double kBacktrackSlope = 0.4;  // CGMethod::BACKTRACKSLOPE
constexpr double kLambdaQuadTol = 1e-3;   // CGMethod::LAMBDAQUADTOL
constexpr int kQuadMaxModels = 100;       // bound on quadraticoptimization's loop
constexpr int kOut = MEDYAN_FF_COUNT + 1;

// Blocks of a vector pass over n3 components. The order of its sums is part of
// a minimization's path: thread t of block b adds components b*256 + t, then
// every blocks*256 after it; a fixed tree adds a block's threads and, in the
// last pass, the blocks.
inline int vec_blocks(int n3) {
    int b = (n3 + kVecThreads - 1) / kVecThreads;
    if (b > 148 * 8) b = 148 * 8;
    return b < 1 ? 1 : b;
}

// ---------------------------------------------------------------- scalars
__device__ __forceinline__ double dmin_ref(double a, double b) { return (b < a) ? b : a; }  // std::min
__device__ __forceinline__ double dmax_ref(double a, double b) { return (a < b) ? b : a; }  // std::max

__device__ void fill_pass(CGState& s, LambdaSet& L) {
    int k = 0;
    if (s.need_e0) L.lam[k++] = 0.0;
    const int want = (s.ls_first_pass && !s.full_passes) ? max(1, s.last_backtracks + 1) : kMaxLambda;
    double lam = s.lam_next;
    int trials = 0;
    while (k < kMaxLambda && trials < want) {
        L.lam[k++] = lam;
        ++trials;
        lam *= 0.5;
        if (lam <= 0.0 || lam <= kLambdaTol) break;  // a further trial would already be a failure
    }
    L.K = k;
    s.k_trials = trials;
}

// Start of a line search (CGMethod.hpp:1316-1324 and :238-262).
__device__ void begin_line_search(CGState& s, LambdaSet& L) {
    s.num_iter++;
    s.ls_active = 1;
    s.ls_first_pass = 1;
    s.backtracks = 0;
    s.skip_force = 1;
    s.move_kind = 0;
    s.reduced_slope = (s.safe_mode ? 0.0 : kBacktrackSlope) * s.slope;
    // QUADRATIC: quadraticLineSearchV2, except in safe mode (CGMethod.hpp:1322-1324)
    s.q_mode = s.ls_quad && !s.safe_mode;
    s.q_phase = 0;
    s.q_maxe = -__builtin_inf();
    s.spec_skip = 1;
    s.spec_valid = 0;
    if (s.grad_inf_norm == 0.0) {  // "return zero if no forces": lambda 0, no energy call
        s.ls_immediate_fail = 1;
        L.K = 0;
        return;
    }
    s.lam_next = dmin_ref(s.lambda_max, s.max_dist / s.grad_inf_norm);
    // speculative force at the first trial, when the previous line search
    // took its first trial (read only by the single-network minimizer)
    if (s.last_backtracks == 0) {
        s.spec_lam = s.lam_next;
        s.spec_skip = 0;
        s.spec_valid = 1;
        s.spec_status = 0;
    }
    fill_pass(s, L);
}

// Line search returned lambda = 0 (CGMethod.hpp:1337-1367).
__device__ void line_search_failed(CGState& s) {
    if (!s.try_to_recover) {
        s.error_flags |= 1;
        s.status = MEDYAN_ERR_LINE_SEARCH;
        s.done = 1;
        s.skip_force = 1;
        return;
    }
    if (s.safe_mode) {
        // funcRecoveryOnError: step = min over coordinates of maxDist/|d_i|
        // = maxDist / max|d_i| (division is monotone), then reset, safe mode off.
        if (!(s.dmax > 0.0)) {
            s.status = MEDYAN_ERR_NONFINITE;  // the reference throws "Invalid step size"
            s.done = 1;
            s.skip_force = 1;
            return;
        }
        s.lam_move = s.max_dist / s.dmax;
        s.move_kind = 2;
        s.skip_force = 0;
    } else {
        s.skip_force = 1;  // resetCGParams, safe mode on; no new force needed
        s.move_kind = 0;
        s.dir_mode = 1;
        s.safe_mode = 1;
    }
}

// End of a quadratic line search with step lq (CGMethod.hpp:637-649):
// lambda = 0 below LAMBDATOL; TotalEnergy and newEnergy stay the
// backtracking energy. The energy at the new point is evaluated at the start
// of the next line search (need_e0), since lq was not the accepted trial.
__device__ void quad_finish(CGState& s, LambdaSet& L, double lq) {
    const double lam = (lq <= 0.0 || lq <= kLambdaTol) ? 0.0 : lq;
    s.q_phase = 0;
    s.ls_active = 0;
    s.last_backtracks = s.backtracks;
    L.K = 0;
    s.total_energy = lam > 0 ? s.q_ebt : s.E_cur;
    if (lam == 0.0) {
        line_search_failed(s);
        return;
    }
    s.lam_move = lam;
    s.E_new = s.q_ebt;
    s.move_kind = 1;
    s.skip_force = 0;
    s.q_used = 1;
}

// One model of quadraticoptimization (CGMethod.hpp:662-714): the parabola
// through (x0,y0), (x1,y1), (x2,y2) and its vertex lq; either the search ends
// or the next pass evaluates E(x + lq*d). The reference's loop has no bound;
// after kQuadMaxModels models it returns x1 here.
__device__ void quad_model(CGState& s, LambdaSet& L) {
    if (s.q_iter >= kQuadMaxModels) {
        quad_finish(s, L, s.q_x1);
        return;
    }
    s.q_iter++;
    const double x0 = s.q_x0, x1 = s.q_x1, x2 = s.q_x2, y0 = s.q_y0, y1 = s.q_y1, y2 = s.q_y2;
    const double d = __dmul_rn(__dmul_rn(__dsub_rn(x0, x1), __dsub_rn(x0, x2)), __dsub_rn(x1, x2));
    const double a = __dadd_rn(__dsub_rn(__dmul_rn(y0, __dsub_rn(x1, x2)), __dmul_rn(y1, __dsub_rn(x0, x2))),
                               __dmul_rn(y2, __dsub_rn(x0, x1)));
    const double t0 = __dmul_rn(__dmul_rn(y0, __dadd_rn(x1, x2)), __dsub_rn(x1, x2));
    const double t1 = __dmul_rn(__dmul_rn(y1, __dadd_rn(x0, x2)), __dsub_rn(x0, x2));
    const double t2 = __dmul_rn(__dmul_rn(y2, __dadd_rn(x0, x1)), __dsub_rn(x0, x1));
    const double b = -__dadd_rn(__dsub_rn(t0, t1), t2);
    const double lq = -b / __dmul_rn(2.0, a);
    if (fabs(__dsub_rn(lq, x1)) / x1 < kLambdaQuadTol) {  // lambda converged
        quad_finish(s, L, lq);
        return;
    }
    if (a / d < 0) {  // no minimum: the backtracking lambda
        quad_finish(s, L, s.q_bt);
        return;
    }
    s.q_lq = lq;
    L.K = 1;
    L.lam[0] = lq;
    s.k_trials = 1;
}

// Energy at the pending quadratic point (CGMethod.hpp:716-763): accept, or
// replace one of the three points and build the next model.
__device__ void quad_eval(CGState& s, LambdaSet& L, double eq) {
    s.num_energy_call++;
    const double lq = s.q_lq, x1 = s.q_x1, y1 = s.q_y1;
    if (fabs(__dsub_rn(eq, y1)) / y1 < kLambdaQuadTol) {
        quad_finish(s, L, lq);
        return;
    }
    if (lq < x1) {
        if (eq < s.q_y0 && eq < y1) {
            s.q_x1 = lq;
            s.q_y1 = eq;
        } else {
            s.q_x0 = lq;
            s.q_y0 = eq;
        }
    } else if (x1 < lq) {
        if (eq < y1 && eq < s.q_y2) {
            s.q_x1 = lq;
            s.q_y1 = eq;
        } else {
            s.q_x2 = lq;
            s.q_y2 = eq;
        }
    } else {  // "Lambda out of range": the previous model's x1
        quad_finish(s, L, x1);
        return;
    }
    quad_model(s, L);
}

// After an energy pass: the reference's backtracking loop over the evaluated
// trial lambdas (CGMethod.hpp:264-362), or the backtracking phase of
// quadraticLineSearchV2 (:564-629) with its trial history, or one
// quadratic-optimization point.
__device__ void ls_decide(CGState& s, LambdaSet& Lr, const double* __restrict__ out) {
    LambdaSet* L = &Lr;
    s.reset_after_dir = 0;
    if (s.done || !s.ls_active) {
        L->K = 0;
        return;
    }
    if (s.ls_immediate_fail) {
        s.ls_immediate_fail = 0;
        s.ls_active = 0;
        s.last_backtracks = 0;
        line_search_failed(s);
        L->K = 0;
        return;
    }
    int slot = 0;
    if (s.need_e0) {
        s.E_cur = out[kOut - 1];
        s.need_e0 = 0;
        slot = 1;
    }
    if (s.q_phase) {
        quad_eval(s, *L, out[kOut - 1]);
        return;
    }
    if (s.ls_first_pass) {
        s.num_energy_call++;  // currentEnergy = energyFunc(coord)
        s.ls_first_pass = 0;
    }
    for (; slot < L->K; ++slot) {
        double lam = L->lam[slot];
        double E_lam = out[slot * kOut + kOut - 1];
        s.num_energy_call++;
        // idealEnergyChange: -(slope*d.F)*lambda (backtracking), -slope*lambda*d.F (V2)
        const double ideal = s.q_mode ? (-kBacktrackSlope * lam) * s.slope : -s.reduced_slope * lam;
        bool decided = false;
        if (lam < 0 || ideal > 0) {  // V2 exits the program here; both end with lambda = 0
            decided = true;
            lam = 0.0;
        }
        const double dE = E_lam - s.E_cur;
        if (dE <= ideal) decided = true;
        else {
            if (s.q_mode) {  // lambdavec/energyvec: the first trial, and the failed ones after it
                if (s.backtracks == 0) {
                    s.q_x2 = lam;
                    s.q_y2 = E_lam;
                } else if (E_lam > s.q_maxe) {
                    s.q_maxe = E_lam;
                }
            }
            lam *= 0.5;
        }
        if (lam <= 0.0 || lam <= kLambdaTol) {
            decided = true;
            lam = 0.0;
            E_lam = s.E_cur;
        }
        if (decided) {
            s.total_energy = E_lam;
            s.ls_active = 0;
            s.last_backtracks = s.backtracks;
            L->K = 0;
            if (lam == 0.0) {
                line_search_failed(s);
            } else if (s.q_mode && s.backtracks > 0 && E_lam < s.E_cur && s.q_maxe > E_lam) {
                // quadratic optimization through (0, E0), (lambda, E), (first lambda, its E)
                s.ls_active = 1;
                s.q_phase = 1;
                s.q_iter = 0;
                s.q_x0 = 0.0;
                s.q_y0 = s.E_cur;
                s.q_x1 = lam;
                s.q_y1 = E_lam;
                s.q_bt = lam;
                s.q_ebt = E_lam;
                quad_model(s, *L);
            } else {
                s.lam_move = lam;
                s.E_new = E_lam;
                s.move_kind = 1;
                s.skip_force = 0;
            }
            return;
        }
        s.backtracks++;
        s.lam_next = lam;
    }
    fill_pass(s, *L);  // undecided: evaluate the next halvings
}

// Scalar part of the dots pass (one thread): F.F = a, F.Fprev = b, max|F| = m.
__device__ void dots_tail(CGState& s, double a, double b, double m) {
    s.num_force_call++;
    s.grad_inf_norm = m;  // maxF (CGMethod.hpp:202-212)
    if (isinf(m)) {
        s.status = MEDYAN_ERR_NONFINITE;  // "maxF is infinity"
        s.done = 1;
    }
    s.new_grad = a;
    s.prev_grad = b;
    if (s.move_kind == 1) {
        s.energy_rel_change = fabs(s.E_new - s.prev_energy) / fabs(s.prev_energy);
        s.prev_energy = s.E_new;
        s.E_cur = s.E_new;
        s.need_e0 = s.q_used;  // a quadratic step moved to a point whose energy is not known
        s.q_used = 0;
        if (s.method == MEDYAN_CG_POLAK_RIBIERE) s.beta = dmax_ref(0.0, (s.new_grad - s.prev_grad) / s.last_fdotf);
        else if (s.method == MEDYAN_CG_FLETCHER_RIEVES) s.beta = s.new_grad / s.last_fdotf;
        else s.beta = 0.0;
        s.dir_mode = 0;
        // copycoordsifminimumE (CGMethod.hpp:1564-1566)
        s.copy_min_e = 0;
        if (m <= 10 * s.grad_tol && s.num_iter > s.force_call_limit / 2 && s.total_energy <= s.min_e) {
            s.min_e = s.total_energy;
            s.copy_min_e = 1;
            s.have_min_e = 1;
        }
    } else {
        // setup (move_kind 0) or recovery step (2): resetCGParams follows
        if (s.move_kind == 2) {
            s.need_e0 = 1;
            s.safe_mode = 0;
        }
        s.dir_mode = 1;
        s.copy_min_e = 0;
    }
    s.parity ^= 1;
    s.skip_force = 1;
}

// Scalar part of the direction pass (one thread): d.F = a, max|d| = m.
__device__ void dir_tail(CGState& s, LambdaSet& L, double a, double m) {
    s.copy_min_e = 0;
    s.dmax = m;
    if (s.dir_mode == 0 && a <= 0) {
        // conjugacy lost: resetCGParams (d = F; its d.F is F.F)
        s.reset_after_dir = 1;
        s.slope = s.new_grad;
        s.dmax = s.grad_inf_norm;
    } else {
        s.slope = a;
    }
    if (s.method != MEDYAN_CG_STEEPEST) s.last_fdotf = s.new_grad;
    s.dir_mode = 0;
    // loop condition (CGMethod.hpp:1279-1282)
    const bool limit = (s.energy_call_limit != 0 && s.num_energy_call > s.energy_call_limit) ||
                       (s.force_call_limit != 0 && s.num_force_call > s.force_call_limit);
    const bool conv = s.grad_inf_norm < s.grad_tol || s.energy_rel_change < s.energy_rel_tol;
    if (limit || conv) {
        s.done = 1;
        s.call_limit = limit;
        L.K = 0;
    } else {
        begin_line_search(s, L);
    }
}

}  // namespace
}  // namespace mb
