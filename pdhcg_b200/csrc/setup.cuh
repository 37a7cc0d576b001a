// setup.cuh -- device preprocessing: transposition, rescaling, starting
// point, power method.  Rescaling restates the reference's host code
// (src/preconditioner.c:256-713) operation for operation so that Ruiz and
// Pock-Chambolle factors are bit-identical: per-row maxima and sums run
// sequentially in CSR order, per-column ones sequentially over the rows of
// A^T (increasing row index, the order of the reference's scatter loop).
#pragma once

#include <cooperative_groups.h>

#include "gridsum.cuh"
#include "kernels.cuh"

namespace pdhcg {

namespace cg = cooperative_groups;

// Row-wise set-up kernels run one thread per row.  With skip_long set, rows
// of more than LONG_ROW entries are skipped and left to the companion
// kernel over the long-row table, one block per long row, so that a dense
// row does not hold one thread for its whole length.

__global__ void expand_rows_kernel(const int *rp, int rows, int *row_of, int skip_long)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        if (skip_long && rp[r + 1] - rp[r] > LONG_ROW)
            continue;
        for (int k = rp[r]; k < rp[r + 1]; ++k)
            row_of[k] = r;
    }
}

__global__ void expand_long_rows_kernel(LongRows L, const int *rp, int *row_of)
{
    for (int i = blockIdx.x; i < L.n; i += gridDim.x) {
        const int r = L.rows[i];
        for (int k = rp[r] + threadIdx.x; k < rp[r + 1]; k += blockDim.x)
            row_of[k] = r;
    }
}

// fixed-order block reductions of one value per thread (blockDim.x == TPB)
__device__ __forceinline__ double block_sum_fixed(double v)
{
    __shared__ double sh[TPB];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = TPB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

__device__ __forceinline__ double block_max(double v)
{
    __shared__ double sh[TPB];
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = TPB / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + o]);
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

// bad != 0 unless the CSR holds exactly the columns 0..cols-1 in order in every row
__global__ void dense_rows_check_kernel(int rows, int cols, const int *rp, const int *ci, int *bad)
{
    const long long nnz = (long long)rows * cols;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nnz;
         k += (long long)gridDim.x * blockDim.x) {
        if (ci[k] != (int)(k % cols))
            atomicOr(bad, 1);
        if (k <= rows && rp[k] != (int)(k * cols)) // row pointers (rows + 1 <= nnz + 1 entries)
            atomicOr(bad, 1);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && rp[rows] != (int)nnz)
        atomicOr(bad, 1);
}

// *flag = 1 when an entry of v[0, n) is NaN (strict = 0: bounds, where
// +-inf means "no bound") or not finite (strict = 1: objective, matrices)
__global__ void nonfinite_kernel(const double *v, long long n, int strict, int *flag)
{
    bool bad = false;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double x = v[i];
        bad |= strict ? !isfinite(x) : isnan(x);
    }
    if (__any_sync(FULL, bad) && (threadIdx.x & 31) == 0)
        atomicOr(flag, 1);
}

__global__ void iota_kernel(int *v, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[i] = i;
}

// rp_t[c] = first position of key >= c in the sorted column keys
__global__ void col_ptr_kernel(const int *keys, int nnz, int ncols, int *rp_t)
{
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncols; c += gridDim.x * blockDim.x) {
        int lo = 0, hi = nnz;
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (keys[mid] < c)
                lo = mid + 1;
            else
                hi = mid;
        }
        rp_t[c] = lo;
    }
}

__global__ void gather_transpose_kernel(const int *perm, const int *row_of, const double *val, int nnz, int *ci_t,
                                        double *v_t)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x) {
        int p = perm[k];
        ci_t[k] = row_of[p];
        v_t[k] = val[p];
    }
}

__global__ void row_absmax_kernel(const int *rp, const double *v, int rows, double *out, int skip_long)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        if (skip_long && rp[r + 1] - rp[r] > LONG_ROW)
            continue;
        double mx = 0.0;
        for (int k = rp[r]; k < rp[r + 1]; ++k) {
            double a = fabs(v[k]);
            if (a > mx)
                mx = a;
        }
        out[r] = mx;
    }
}

// Long rows of the set-up passes: one block per row, or one warp where the
// rows are short of a block's width (2e5 rows of 102 entries: 340 us a pass
// with a block per row, whose reduction outweighs the row).
constexpr int LONG_WARP_MEAN = 1024; // mean entries up to which a warp takes a row

// f(row, first lane, lanes) for every long row; WARP: a warp per row
template <bool WARP, typename F>
__device__ __forceinline__ void for_long_rows(const LongRows &L, F &&f)
{
    if (WARP) {
        const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
        for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < L.n; i += nw)
            f(L.rows[i], lane, 32);
    } else {
        for (int i = blockIdx.x; i < L.n; i += gridDim.x)
            f(L.rows[i], (int)threadIdx.x, (int)blockDim.x);
    }
}

// the maximum is exact in any order, so a long row's value is the same
template <bool WARP>
__global__ void long_row_absmax_kernel(LongRows L, const int *rp, const double *v, double *out)
{
    for_long_rows<WARP>(L, [&](int r, int at, int step) {
        double mx = 0.0;
#pragma unroll 4
        for (int k = rp[r] + at; k < rp[r + 1]; k += step)
            mx = fmax(mx, fabs(v[k]));
        mx = WARP ? warp_max(mx) : block_max(mx);
        if (at == 0)
            out[r] = mx;
    });
}

// sum_k |a_k|^p per row; p == 1 uses |a| itself (pow(x, 1) == x exactly)
__global__ void row_powsum_kernel(const int *rp, const double *v, int rows, double p, double *out, int skip_long)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        if (skip_long && rp[r + 1] - rp[r] > LONG_ROW)
            continue;
        double s = 0.0;
        for (int k = rp[r]; k < rp[r + 1]; ++k) {
            double a = fabs(v[k]);
            s += (p == 1.0) ? a : pow(a, p);
        }
        out[r] = s;
    }
}

// a long row's sum in a fixed order (thread-strided, then a tree): the same
// on every run, but associated differently from a sequential sum
template <bool WARP>
__global__ void long_row_powsum_kernel(LongRows L, const int *rp, const double *v, double p, double *out)
{
    for_long_rows<WARP>(L, [&](int r, int at, int step) {
        double t = 0.0;
#pragma unroll 4
        for (int k = rp[r] + at; k < rp[r + 1]; k += step) {
            const double a = fabs(v[k]);
            t += (p == 1.0) ? a : pow(a, p);
        }
        t = WARP ? warp_sum(t) : block_sum_fixed(t);
        if (at == 0)
            out[r] = t;
    });
}

__global__ void sqrt_or_one_kernel(double *v, int n)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[i] = v[i] < 1e-12 ? 1.0 : sqrt(v[i]);
}

// Cone-preserving aggregation of a scaling vector over each cone block
// (reference apply_cone_scaling_adjustment, src/preconditioner.c:108-144).
__global__ void cone_scaling_adjust_kernel(double *s, int ncones, const int *start, const int *len, int ruiz_phase)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < ncones; b += gridDim.x * blockDim.x) {
        int st = start[b], L = len[b];
        double mx = 0.0, sq = 0.0;
        for (int i = st; i < st + L; ++i) {
            mx = fmax(mx, s[i]);
            sq += s[i] * s[i];
        }
        double rms = sqrt(sq / (double)L);
        double bs = ruiz_phase ? (L <= 8 ? mx : rms) : (L <= 8 ? rms : sqrt(mx * rms));
        for (int i = st; i < st + L; ++i)
            s[i] = bs;
    }
}

// Diagonal-congruence projection of the log scaling of a PSD block, used
// when cone-preserving scaling is off (reference project_psd_log_scaling,
// src/preconditioner.c:46-92); one thread per block, order <= 64.
// log_space: s already holds log scales (Curtis-Reid) and receives log scales
__global__ void psd_scaling_kernel(double *s, int ncones, const int *start, const int *vdim, const int *type,
                                   int log_space)
{
    const double LIM = 69.07755278982137;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < ncones; b += gridDim.x * blockDim.x) {
        if (type[b] != 4)
            continue;
        int st = start[b], order = vdim[b];
        if (order > 64)
            continue;
        double f[64];
        for (int i = 0; i < order; ++i)
            f[i] = 0.0;
        int slot = st;
        for (int col = 0; col < order; ++col)
            for (int row = col; row < order; ++row, ++slot) {
                double v = log_space ? s[slot] : log(fmax(s[slot], 1e-300));
                if (isnan(v))
                    v = 0.0;
                else if (v > LIM)
                    v = LIM;
                else if (v < -LIM)
                    v = -LIM;
                if (row == col)
                    f[row] += 2.0 * v;
                else {
                    f[row] += v;
                    f[col] += v;
                }
            }
        double rhs = 0.0;
        for (int i = 0; i < order; ++i)
            rhs += f[i];
        double corr = rhs / (2.0 * order + 2.0), diag = order + 2.0;
        for (int i = 0; i < order; ++i) {
            f[i] = (f[i] - corr) / diag;
            f[i] = fmax(-0.5 * LIM, fmin(0.5 * LIM, f[i]));
        }
        slot = st;
        for (int col = 0; col < order; ++col)
            for (int row = col; row < order; ++row, ++slot)
                s[slot] = log_space ? f[row] + f[col] : exp(f[row] + f[col]);
    }
}

// v_k /= (rs[r] * cs[col]) : A with (cr, vr), A^T with (vr, cr), Q with (vr, vr)
__global__ void scale_csr_kernel(const int *rp, const int *ci, double *v, int rows, const double *rs,
                                 const double *cs, int cr_first, int skip_long)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        if (skip_long && rp[r + 1] - rp[r] > LONG_ROW)
            continue;
        double a = rs[r];
        for (int k = rp[r]; k < rp[r + 1]; ++k) {
            double b = cs[ci[k]];
            v[k] /= cr_first ? (b * a) : (a * b);
        }
    }
}

template <bool WARP>
__global__ void long_scale_csr_kernel(LongRows L, const int *rp, const int *ci, double *v, const double *rs,
                                      const double *cs, int cr_first)
{
    for_long_rows<WARP>(L, [&](int r, int at, int step) {
        const double a = rs[r];
#pragma unroll 4
        for (int k = rp[r] + at; k < rp[r + 1]; k += step) {
            const double b = cs[ci[k]];
            v[k] /= cr_first ? (b * a) : (a * b);
        }
    });
}

// v_k /= rs[r] for every entry of row r (rows of at most LONG_ROW entries:
// every caller's matrix has none longer)
__global__ void scale_rows_kernel(const int *rp, double *v, int rows, const double *rs)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        double a = rs[r];
        for (int k = rp[r]; k < rp[r + 1]; ++k)
            v[k] /= a;
    }
}

// v_k /= cs[ci[k]], one thread per entry (no row needed)
__global__ void scale_cols_kernel(const int *ci, double *v, long long nnz, const double *cs)
{
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nnz;
         k += (long long)gridDim.x * blockDim.x)
        v[k] /= cs[ci[k]];
}

__global__ void scale_vectors_kernel(int n, int m, double *c, double *l, double *u, const double *vr, double *lc,
                                     double *uc, double *g, const double *cr, double *cum_vr, double *cum_cr)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
        if (i < n) {
            c[i] /= vr[i];
            u[i] *= vr[i];
            l[i] *= vr[i];
            cum_vr[i] *= vr[i];
        } else {
            int r = i - n;
            lc[r] /= cr[r];
            uc[r] /= cr[r];
            g[r] /= cr[r];
            cum_cr[r] *= cr[r];
        }
    }
}

__global__ void mul_scalar_kernel(double *v, int n, double f)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[i] *= f;
}

// squares for the bound / objective rescaling norms (reference bound_obj_rescaling,
// src/preconditioner.c:602-652) and max/sq for the unscaled relative-error norms
// (src/solver_state.cu:854-934)
enum NormScalar { NS_B2 = 0, NS_C2, NS_BMAX, NS_CMAX, NS_COUNT };

__global__ void __launch_bounds__(TPB) norms_kernel(int n, int m, const double *c, const double *lc, const double *uc,
                                                    const double *g, double *partials)
{
    const int ops[NS_COUNT] = {RSUM, RSUM, RMAX, RMAX};
    double acc[NS_COUNT] = {0.0, 0.0, 0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
        if (i < n) {
            double v = c[i];
            acc[NS_C2] += v * v;
            acc[NS_CMAX] = fmax(acc[NS_CMAX], fabs(v));
        } else {
            int r = i - n;
            double lo = lc[r], up = uc[r], gg = g[r];
            double b2 = 0.0, bm = fabs(gg);
            if (isfinite(lo) && lo != up) {
                b2 += lo * lo;
                bm = fmax(bm, fabs(lo));
            }
            if (isfinite(up)) {
                b2 += up * up;
                bm = fmax(bm, fabs(up));
            }
            acc[NS_B2] += b2 + gg * gg;
            acc[NS_BMAX] = fmax(acc[NS_BMAX], bm);
        }
    }
    block_reduce_store<NS_COUNT>(acc, ops, partials);
}

__global__ void bound_obj_scale_kernel(int n, int m, double sb, double sc, double *c, double *l, double *u, double *lc,
                                       double *uc, double *g)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
        if (i < n) {
            l[i] *= sb;
            u[i] *= sb;
            c[i] *= sc;
        } else {
            int r = i - n;
            lc[r] *= sb;
            uc[r] *= sb;
            g[r] *= sb;
        }
    }
}

// diagonal of a diagonal-only Q, plus the reference's 1e-12
// (preprocess_qp_problem, src/preconditioner.c:812-825)
__global__ void q_diag_kernel(const int *rp, const int *ci, const double *v, int n, double *qd)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        for (int k = rp[r]; k < rp[r + 1]; ++k)
            if (ci[k] < n)
                qd[ci[k]] = v[k] + 1e-12;
}

// starting point: warm start scaling, cone interior aux points, box clamp
// (reference initialize_solver_state / initialize_cone_runtime,
// src/solver_state.cu:578-686, 809-829, 983-1000)
__global__ void scale_start_kernel(int n, const double *start, const double *vr, double sb, double *x0)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        x0[i] = start[i] * vr[i] * sb;
}

// fixed: slots fixed by set_cone_fixed (NULL: none), which keep their value
__global__ void cone_aux_init_kernel(int ncones, const int *start, const int *vdim, const int *type,
                                     const double *vr, double sb, double *x0, const unsigned char *fixed)
{
    const double INV_SQRT2 = 0.7071067811865475;
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < ncones; b += gridDim.x * blockDim.x) {
        int aux0 = start[b] + vdim[b];
        if (type[b] == 1) { // standard SOC: w, z
            if (!(fixed && fixed[aux0]))
                x0[aux0] = -INV_SQRT2 * sb * vr[aux0];
            if (!(fixed && fixed[aux0 + 1]))
                x0[aux0 + 1] = INV_SQRT2 * sb * vr[aux0 + 1];
        } else if (type[b] == 0) { // rotated SOC: t
            if (!(fixed && fixed[aux0 + 1]))
                x0[aux0 + 1] = sb * vr[aux0 + 1];
        }
    }
}

// fixed cone slots: the scaled bounds pinned at value * vr * sb (reference
// pin_scaled_fixed_cone_bounds, src/preconditioner.c:311-327)
__global__ void pin_fixed_kernel(int nfix, const int *idx, const double *val, const double *vr, double sb, double *l,
                                 double *u)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nfix; k += gridDim.x * blockDim.x) {
        const int j = idx[k];
        const double v = val[k] * vr[j] * sb;
        l[j] = v;
        u[j] = v;
    }
}

__global__ void box_clamp_copy_kernel(int n, const double *l, const double *u, double *x0, double *x, double *xp,
                                      double *xr)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double v = fmax(l[i], fmin(x0[i], u[i]));
        x0[i] = v;
        x[i] = v;
        xp[i] = v;
        xr[i] = v;
    }
}

__global__ void dual_start_kernel(int m, const double *start, const double *cr, double sc, double *y0, double *y,
                                  double *yp)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
        double v = start ? start[i] * cr[i] * sc : 0.0;
        y0[i] = v;
        y[i] = v;
        yp[i] = v;
    }
}

// restart: x_init = x_cur = x_pdhg, y_init = y_cur = y_pdhg
template <typename VT>
__global__ void restart_copy_kernel(int n, int m, const VT *xp, VT *x0, VT *x, const VT *yp, VT *y0, VT *y)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
        if (i < n) {
            VT v = xp[i];
            x0[i] = v;
            x[i] = v;
        } else {
            int r = i - n;
            VT v = yp[r];
            y0[r] = v;
            y[r] = v;
        }
    }
}

// Final answer: reduced cost and unscaling (reference create_result_from_state
// and compute_and_rescale_reduced_cost_qp_kernel, src/pdhg_core_op.cu:1431-1471,
// src/kernels/pdhcg_kernels.cu:866-894, rescale_solution_kernel :308-327).
template <typename VT>
__global__ void result_kernel(int n, int m, const int *At_rp, const int *At_ci, const double *At_v, const double *c,
                              const double *q, const double *qx, int qmode, const double *l, const double *u,
                              const double *vr, const double *cr, double sb, double sc, const VT *xp,
                              const VT *yp, double *x_out, double *y_out, double *rc_out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n + m; i += gridDim.x * blockDim.x) {
        if (i < n) {
            double aty = row_dot<1>(At_rp, At_ci, At_v, yp, i, 0);
            double g = c[i];
            if (qmode == 1)
                g += q[i] * (double)xp[i];
            else if (qmode == 2)
                g += qx[i];
            double rc = (g - aty) * vr[i] / sc;
            if (!isfinite(l[i]))
                rc = fmin(rc, 0.0);
            if (!isfinite(u[i]))
                rc = fmax(rc, 0.0);
            rc_out[i] = rc;
            x_out[i] = (double)xp[i] / vr[i] / sb;
        } else {
            int r = i - n;
            y_out[r] = (double)yp[r] / cr[r] / sc;
        }
    }
}

// ---------------------------------------------------------------------------
// Lanczos process of A A^T (m x m) for the step size, `steps` more steps in
// one cooperative launch.  Vectors are kept unnormalised with their scale
// (q_j = inv u_j); a step is
//   z = A^T q_j;  alpha_j = |z|^2;
//   u_{j+1} = A z - beta_{j-1} q_{j-1} - alpha_j q_j  (over u_{j-1});
//   beta_j = |u_{j+1}|
// with two grid-wide sums, which are also its barriers.  One block of 32
// warps per SM (fewer on small problems: the barrier's cost grows with the
// blocks).
// ---------------------------------------------------------------------------
constexpr int LANCZOS_MAX = 512, LANCZOS_CHUNK = 16, LANCZOS_TPB = 1024;
constexpr int LANCZOS_SMEM = (LANCZOS_TPB / 32) * STREAM_CHUNK * (int)sizeof(double);

struct LanczosData {
    int m, n;
    const int *A_rp, *A_ci;
    const double *A_v;
    const int *At_rp, *At_ci;
    const double *At_v;
    LongRows A_long, At_long;
    double *u[2]; // the start vector in u[0]
    double *z;
    double *out; // [0] inv of the current vector, [1] inv of the previous, [2] beta between them,
                 // [3] steps done, then alpha[LANCZOS_MAX], beta[LANCZOS_MAX]
};

static __global__ void __launch_bounds__(LANCZOS_TPB) lanczos_kernel(LanczosData L, GridSlots S, int j0, int steps)
{
    extern __shared__ double lanczos_stage[];
    __shared__ double sh[LANCZOS_TPB / 32 + 1];
    const int NW = LANCZOS_TPB / 32;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = blockIdx.x * NW + wib, nw = gridDim.x * NW;
    double *stage = lanczos_stage + wib * STREAM_CHUNK;
    double inv, inv_prev = 0.0, beta = 0.0;
    grid_begin(S);
    if (j0 == 0) {
        double a = 0.0;
        for (int i = blockIdx.x * LANCZOS_TPB + threadIdx.x; i < L.m; i += gridDim.x * LANCZOS_TPB)
            a += L.u[0][i] * L.u[0][i];
        inv = 1.0 / sqrt(grid_sum<NW>(a, S, sh));
    } else {
        inv = L.out[0];
        inv_prev = L.out[1];
        beta = L.out[2];
        grid_barrier(S); // every block has read the state that block 0 will write
    }
    int j = j0;
    double last = 0.0; // scale of T, for the exhaustion test
    for (; j < j0 + steps; ++j) {
        double *u = L.u[j & 1], *up = L.u[(j & 1) ^ 1];
        if (L.At_long.n > 0) { // segment pass of the long rows, then the rows
            long_partials<true>(L.At_long, L.At_ci, L.At_v, u, gw, nw, lane);
            grid_barrier(S);
        }
        double a = 0.0;
        for (int t = gw; t < (L.n + 31) / 32; t += nw) {
            const int r0 = 32 * t, nr = min(32, L.n - r0);
            double r[1];
            warp_stream_rows<1, true>(L.At_rp, L.At_ci, L.At_v, u, r0, nr, lane, stage, r, L.At_long);
            if (lane < nr) {
                const double z = r[0] * inv;
                L.z[r0 + lane] = z;
                a += z * z;
            }
        }
        const double alpha = grid_sum<NW>(a, S, sh);
        if (L.A_long.n > 0) {
            long_partials<true>(L.A_long, L.A_ci, L.A_v, L.z, gw, nw, lane);
            grid_barrier(S);
        }
        a = 0.0;
        for (int t = gw; t < (L.m + 31) / 32; t += nw) {
            const int r0 = 32 * t, nr = min(32, L.m - r0);
            double r[1];
            warp_stream_rows<1, true>(L.A_rp, L.A_ci, L.A_v, L.z, r0, nr, lane, stage, r, L.A_long);
            if (lane < nr) {
                const int i = r0 + lane;
                const double prev = j > 0 ? beta * inv_prev * __ldcg(up + i) : 0.0;
                const double w = (r[0] - prev) - alpha * inv * __ldcg(u + i);
                up[i] = w;
                a += w * w;
            }
        }
        const double b = sqrt(grid_sum<NW>(a, S, sh));
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            L.out[4 + j] = alpha;
            L.out[4 + LANCZOS_MAX + j] = b;
        }
        last = fmax(last, alpha);
        if (!(b > 1e-14 * last)) { // the Krylov space is exhausted: T is exact
            ++j;
            break;
        }
        beta = b;
        inv_prev = inv;
        inv = 1.0 / b;
    }
    grid_end(S);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        L.out[0] = inv;
        L.out[1] = inv_prev;
        L.out[2] = beta;
        L.out[3] = (double)j;
    }
}

// ---- Curtis-Reid scaling (reference curtis_reid_rescaling,
// src/preconditioner.c:334-495): log-space alternating row / column averages
// of log|a_ij|, cone blocks averaged together when scaling is
// cone-preserving.  One thread per row with sequential sums in entry order,
// the order of the reference's host loops.
constexpr double CR_LOG_MIN_ABS = 1e-300;
constexpr double CR_LOG_LIMIT = 69.07755278982137; // log(1e30)

// sum of log max(|a|, 1e-300) over each row of M
__global__ void cr_logsum_kernel(const int *rp, const double *v, int rows, double *sum)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int k = rp[r]; k < rp[r + 1]; ++k)
            s += log(fmax(fabs(v[k]), CR_LOG_MIN_ABS));
        sum[r] = s;
    }
}

// raw[r] = base[r] - sum_{k in row r} other[col k]; out[r] = raw[r] / len(r),
// 0 for empty rows (raw may be NULL)
__global__ void cr_average_kernel(const int *rp, const int *ci, int rows, const double *base, const double *other,
                                  double *out, double *raw)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        int b = rp[r], e = rp[r + 1];
        double s = base[r];
        for (int k = b; k < e; ++k)
            s -= other[ci[k]];
        if (raw)
            raw[r] = s;
        out[r] = e > b ? s / (double)(e - b) : 0.0;
    }
}

// cone-preserving column step: one value per cone block,
// (sum over the block of cs) / (sum over the block of the column counts)
__global__ void cr_cone_average_kernel(int nc, const int *start, const int *len, const int *At_rp, const double *cs,
                                       double *cls)
{
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nc; b += gridDim.x * blockDim.x) {
        const int st = start[b], L = len[b];
        double bsum = 0.0;
        int bcount = 0;
        for (int c = st; c < st + L; ++c) {
            bsum += cs[c];
            bcount += At_rp[c + 1] - At_rp[c];
        }
        const double bl = bcount > 0 ? bsum / (double)bcount : 0.0;
        for (int c = st; c < st + L; ++c)
            cls[c] = bl;
    }
}

__global__ void cr_exp_kernel(double *v, int k)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k; i += gridDim.x * blockDim.x) {
        double x = v[i];
        if (isnan(x))
            v[i] = 1.0;
        else
            v[i] = exp(fmin(fmax(x, -CR_LOG_LIMIT), CR_LOG_LIMIT));
    }
}

} // namespace pdhcg
