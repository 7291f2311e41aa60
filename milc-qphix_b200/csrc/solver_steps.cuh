// Scalar steps of the solvers: what follows a reduction, as functors on a
// SolverState.  The reducing kernels (dslash.cu, blas.cu) run them in their
// last block on the device-wide state; the resident solver loop (loop.cu)
// runs them in every block on the block's own copy.
#pragma once

#include <climits>

#include "device_common.cuh"

namespace qb {

// Scalar step after p.(M^dag M p) is known, run by one warp of the last
// block of the reduction: CG (mode 0) a = -rsq/pkp in lane 0; multi-shift
// (mode 1) the shift recurrences, lane k handling shifts k, k + 32, ...
// (each shift's arithmetic is the sequential one, so the results do not
// depend on the lane split; one thread walking the shifts through device
// memory took ~10 us per iteration at 12 shifts).
// A zero or non-finite p.(M p) is a breakdown (M is positive definite for
// m > 0; the reference divides by it unchecked, ks_d_congrad_fn.cpp:511):
// the step is set to zero, st->error = 2 and the update kernel that follows
// ends the device run, so the host returns QPHIX_FAIL.
struct FinMdagm {
    SolverState *st;
    int mode;
    static constexpr bool kWarp = true;
    __device__ void operator()(const double *t, int lane) const
    {
        const double pkp = t[0];
        int done = 0;
        if (lane == 0) {
            st->pkp = pkp;
            st->iteration += 1;
            if (!(pkp != 0.0) || !isfinite(pkp)) {
                st->error = 2;
                st->a = 0.0;
                done = 1;
            } else if (mode == 0) {
                st->a = round_to(-st->rsq / pkp, st->prec_single);
                done = 1;
            }
        }
        if (__shfl_sync(0xffffffffu, done, 0)) return;
        // multi-shift scalar recurrences (ks_multicg_offset.cpp:475-496);
        // the values of the previous iteration are scrolled first
        // (:617-622), which the reference does at the end of that iteration
        const int single = st->prec_single;
        const int jl = st->j_low;
        const int nn = st->num_now;
        if (!st->first_iter) {
            for (int k = lane; k < nn; k += 32) {
                st->beta_im1[k] = st->beta_i[k];
                st->zeta_im1[k] = st->zeta_i[k];
                st->zeta_i[k] = st->zeta_ip1[k];
            }
        }
        __syncwarp();
        if (lane == 0) {
            st->first_iter = 0;
            st->beta_i[jl] = round_to(-st->rsq / pkp, single);
            st->zeta_ip1[jl] = 1.0;
        }
        __syncwarp();
        const double b_jl = st->beta_i[jl], a_jl = st->alpha[jl], bm1_jl = st->beta_im1[jl];
        for (int k = lane; k < nn; k += 32) {
            if (k == jl) continue;
            const double zi = st->zeta_i[k], zim1 = st->zeta_im1[k];
            double z = round_to(round_to(zi * zim1, single) * bm1_jl, single);
            const double c1 = round_to(round_to(b_jl * a_jl, single) * round_to(zim1 - zi, single), single);
            const double c2 =
                round_to(round_to(zim1 * bm1_jl, single) * (1.0 + round_to(st->shifts[k] * b_jl, single)), single);
            const double den = round_to(c1 + c2, single);
            if (den != 0.0) z = round_to(z / den, single);
            else { z = 0.0; st->finished[k] = 1; }
            st->zeta_ip1[k] = z;
            if (zi != 0.0)
                st->beta_i[k] = round_to(round_to(b_jl * z, single) / zi, single);
            else { st->zeta_ip1[k] = 0.0; st->beta_i[k] = 0.0; st->finished[k] = 1; }
        }
        __syncwarp();
        // the last active shift leaves the recurrence once it has finished
        if (lane == 0 && nn - 1 > jl && st->finished[nn - 1] == 1) st->num_now = nn - 1;
    }
};

// calc_rsq2 (ks_d_congrad_fn.cpp:131-147): x += a p; r += a ttt; rsq = |r|^2
// followed by the scalar bookkeeping of :543-566 and the completion test at
// the top of the loop (:360-363), evaluated on the device.
// V: sites of the whole lattice (relative_residue divides by the global
// volume, ks_blas_utils_c.cpp:148)
struct FinCgUpdate {
    SolverState *st;
    int gate;
    bool relres;
    double V;
    __device__ void operator()(const double *t) const
    {
        const int single = st->prec_single;
        const double oldrsq = st->rsq;
        const double rsq = t[0];
        st->oldrsq = oldrsq;
        st->rsq = rsq;
        double relrsq = st->relrsq;
        if (relres) relrsq = round_to(sqrt(2.0 * t[1] / V), single);
        st->relrsq = relrsq;
        st->size_r = round_to(rsq, single) / st->source_norm;
        st->size_relr = round_to(relrsq, single);
        st->b = round_to(round_to(rsq, single) / oldrsq, single);
        const bool conv = (st->rsqmin <= 0 || st->rsqmin > st->size_r) &&
                          (st->relrsqmin <= 0 || st->relrsqmin > st->size_relr);
        if (!isfinite(rsq) && !st->error) st->error = 1;  // non-finite residual: breakdown
        if ((st->iteration % st->niter == 0) || conv || st->error || run_guard(st)) stop_run(st, gate);
    }
};

// end of an inner iteration of the mixed CG (one thread): b, and whether
// to stop for a reliable update
__device__ __forceinline__ void mx_finish(SolverState *st, double rsq, int gate, double delta2)
{
    const double oldrsq = st->rsq;
    st->oldrsq = oldrsq;
    st->rsq = rsq;
    st->b = rsq / oldrsq;
    bool stalled = false;
    if (rsq < st->ru_best) {
        st->ru_best = rsq;
        st->ru_best_iter = st->iteration;
    } else if (st->ru_stall_window > 0 && st->iteration - st->ru_best_iter >= st->ru_stall_window) {
        stalled = true;
        st->ru_stalled = 1;
    }
    if (!isfinite(rsq) && !st->error) st->error = 1;  // non-finite residual: breakdown
    const bool ru = (rsq < delta2 * st->rsq_ru) || (rsq <= st->rsqstop) || stalled ||
                    (st->iteration >= st->max_cg) || st->error || run_guard(st);
    if (ru) {
        st->skip_axpy = 1;  // this iteration's p update waits for the true residual
        stop_run(st, gate);
    }
}

struct FinMx {
    SolverState *st;
    int gate;
    double delta2;
    __device__ void operator()(const double *t) const { mx_finish(st, t[0], gate, delta2); }
};

// calc_rsq2 (ks_multicg_offset.cpp:124-140) + the convergence test (:520)
// + the alpha recurrences (:587-598), evaluated on the device.
struct FinMsResidual {
    SolverState *st;
    int gate;
    // one warp: lane k updates shifts k, k + 32, ... (per-shift arithmetic
    // as in the sequential form)
    static constexpr bool kWarp = true;
    __device__ void operator()(const double *t, int lane) const
    {
        const int single = st->prec_single;
        const double rsq = t[0];
        int done = 0;
        if (lane == 0) {
            const double oldrsq = st->rsq;
            st->oldrsq = oldrsq;
            st->rsq = rsq;
            if (!isfinite(rsq) && !st->error) st->error = 1;  // non-finite residual: breakdown
            if (st->error) {  // (or a zero p.Ap in the Dslash kernel before)
                stop_run(st, gate);
                done = 1;
            } else if (rsq <= st->rsqstop) {
                st->converged = 1;
                stop_run(st, gate);
                done = 1;
            } else {
                st->alpha[st->j_low] = round_to(rsq / oldrsq, single);
            }
        }
        if (__shfl_sync(0xffffffffu, done, 0)) return;
        __syncwarp();
        const int jl = st->j_low;
        const int nn = st->num_now;
        const double a_jl = st->alpha[jl], b_jl = st->beta_i[jl];
        const int it = st->iteration;
        const double stop = st->shift_stop;
        for (int k = lane; k < nn; k += 32) {
            if (k == jl) continue;
            const double zb = round_to(st->zeta_i[k] * b_jl, single);
            if (zb != 0.0)
                st->alpha[k] = round_to(round_to(round_to(a_jl * st->zeta_ip1[k], single) * st->beta_i[k], single) / zb,
                                        single);
            else { st->alpha[k] = 0.0; st->finished[k] = 1; }
            if (stop > 0.0 && st->shift_done_at[k] == INT_MAX) {
                const double z = st->zeta_ip1[k];
                if (z * z * rsq <= stop) st->shift_done_at[k] = it;
            }
        }
        __syncwarp();
        if (lane == 0) {
            // the iteration completes (its vector updates are not gated off);
            // the host then replaces r by the FP64 residual of the base shift
            if (st->ms_delta2 > 0.0 && rsq < st->ms_delta2 * st->rsq_ru) {
                st->ms_ru = 1;
                stop_run(st, gate);
            }
            // deferred shift updates: this iteration takes the segment's last slot
            if (st->ms_seg_cap > 0 && st->iteration - st->ms_seg_start >= st->ms_seg_cap) {
                st->ms_seg_full = 1;
                stop_run(st, gate);
            }
            if (st->iteration >= st->max_cg || run_guard(st)) stop_run(st, gate);
        }
    }
};

}  // namespace qb
