// resident.cuh -- data of the persistent iteration (resident.cu).
#pragma once

#include "device.cuh"

namespace pdhcg {

constexpr int RESIDENT_SLOTS = 10;     // values of the widest grid fold (an evaluation's)
// Iterations of one launch before the host sees the clock and the cancel flag
// again: 6 ms at 2.9 us (300 variables), 16 at 8 (50000), 20 at 10 (150000).
// The launch hands back at its next evaluation point after them.
constexpr int RESIDENT_BUDGET = 2000;

// The loop's scalars, in from the host and back (Solve's members of the same
// meaning).
struct ResidentState {
    double omega, best_omega, best_gap, err_sum, last_err, fpe, fpe0, fpe_last;
    double abs_p, rel_p, abs_d, rel_d, pobj, dobj, gap, rel_gap;
    int k, inner, major, optimal, restarts, evaluations;
    int wait_failed; // out: a grid wait ran out
};

struct ResidentParams {
    int l2, freq, iteration_limit, budget;
    double eps_opt, eps_feas, step, nonconvexity, rho, sb, sc, cnorm, bnorm, obj_const;
    double artificial, sufficient, necessary, k_p, k_i, k_d, i_smooth;
};

struct ResidentData {
    int n, m;
    const int *A_rp, *A_ci, *At_rp, *At_ci;
    const double *A_v, *At_v;
    const double *c, *l, *u, *q, *lc, *uc, *g, *vr, *cr; // q NULL: linear program
    double *x0, *x, *xp, *xr, *dx, *ds, *y0, *y, *yp, *dy;
    ResidentState *state;
};

} // namespace pdhcg
