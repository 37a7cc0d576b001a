// resident.cu -- the main loop of a small or middle-sized problem without
// cones (LP or diagonal Q) in one persistent launch.
//
// What bounds such a solve is not its data, which fits on chip (50000
// variables: 4 MB, read in under 1 us), but the launches: two kernels per
// iteration and, every ten iterations at first, an evaluation of two kernels
// with a copy and a host decision behind them, 12 us per iteration on a problem
// of 300 variables as on one of 50000 (now 2.9 and 8).  Here each block keeps its rows of A
// and of A^T and its part of the vectors in shared memory for the whole
// launch; x_refl and y, which the other blocks gather, go through L2, and two
// grid barriers (gridsum.cuh) end an iteration's two products.  Evaluation,
// restart test, PID primal weight and termination are taken on the device by
// every block alike from the same folded scalars (the decisions of
// Solve::loop in the same order), so the host is needed only for the
// infeasibility certificates (major iterations before 3 *
// termination_evaluation_frequency), the clock and the cancel flag.  A problem
// that fits in one block runs without grid barriers, its exchange vectors in
// shared memory.
#include "launch.cuh"

namespace pdhcg {

constexpr int RT = 512, RWARPS = RT / 32;

__device__ __forceinline__ int resident_print_frequency(int iter)
{
    int step = 10;
    long long threshold = 1000;
    while (iter >= threshold) {
        step *= 10;
        threshold *= 10;
    }
    return step;
}

// ONE: a single block, which gathers x_refl and y from its shared memory
template <bool ONE>
__global__ void __launch_bounds__(RT, 1) resident_kernel(ResidentData D, ResidentParams P, GridSlots S, ResidentPlan L)
{
    extern __shared__ __align__(16) double rsm[];
    __shared__ double sh[RESIDENT_SLOTS * (RWARPS + 1)];
    const int tid = threadIdx.x, nb = gridDim.x;
    const int c0 = (int)((long long)D.n * blockIdx.x / nb), c1 = (int)((long long)D.n * (blockIdx.x + 1) / nb);
    const int w0 = (int)((long long)D.m * blockIdx.x / nb), w1 = (int)((long long)D.m * (blockIdx.x + 1) / nb);
    const int nv = c1 - c0, nr = w1 - w0;
    // shared memory: values, vectors, row pointers, indices
    double *p = rsm;
    auto take = [&](int k) {
        double *r = p;
        p += k;
        return r;
    };
    double *tv = take(L.cap_at), *av = take(L.cap_a);
    double *c = take(L.vars), *lo = take(L.vars), *hi = take(L.vars), *q = take(L.vars), *x0 = take(L.vars),
           *x = take(L.vars);
    double *lc = take(L.rows), *uc = take(L.rows), *gg = take(L.rows), *y0 = take(L.rows), *y = take(L.rows);
    double *xrs = take(ONE ? L.vars : 0);
    int *trp = (int *)p, *arp = trp + L.vars + 1, *tci = arp + L.rows + 1, *aci = tci + L.cap_at;
    const int tb = D.At_rp[c0], te = D.At_rp[c1], ab = D.A_rp[w0], ae = D.A_rp[w1];
    for (int k = tid; k < te - tb; k += RT) {
        tv[k] = D.At_v[tb + k];
        tci[k] = D.At_ci[tb + k];
    }
    for (int k = tid; k < ae - ab; k += RT) {
        av[k] = D.A_v[ab + k];
        aci[k] = D.A_ci[ab + k];
    }
    for (int j = tid; j <= nv; j += RT)
        trp[j] = D.At_rp[c0 + j] - tb;
    for (int i = tid; i <= nr; i += RT)
        arp[i] = D.A_rp[w0 + i] - ab;
    for (int j = tid; j < nv; j += RT) {
        c[j] = D.c[c0 + j];
        lo[j] = D.l[c0 + j];
        hi[j] = D.u[c0 + j];
        q[j] = D.q ? D.q[c0 + j] : 0.0;
        x0[j] = D.x0[c0 + j];
        x[j] = D.x[c0 + j];
    }
    for (int i = tid; i < nr; i += RT) {
        lc[i] = D.lc[w0 + i];
        uc[i] = D.uc[w0 + i];
        gg[i] = D.g[w0 + i];
        y0[i] = D.y0[w0 + i];
        y[i] = D.y[w0 + i];
    }
    // row r's product with v, the entries in order, eight gathers in flight
    auto dot = [](const double *sv, const int *sc, int b, int e, const double *v, bool shared) {
        double s = 0.0;
        auto ldv = [&](const double *a) { return shared ? *a : __ldcg(a); };
        int k = b;
        for (; k + 8 <= e; k += 8) {
            double a[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                a[u] = ldv(v + sc[k + u]);
#pragma unroll
            for (int u = 0; u < 8; ++u)
                s += sv[k + u] * a[u];
        }
        if (k + 4 <= e) {
            const double a0 = ldv(v + sc[k]), a1 = ldv(v + sc[k + 1]), a2 = ldv(v + sc[k + 2]),
                         a3 = ldv(v + sc[k + 3]);
            s += sv[k] * a0;
            s += sv[k + 1] * a1;
            s += sv[k + 2] * a2;
            s += sv[k + 3] * a3;
            k += 4;
        }
        const bool p0 = k < e, p1 = k + 1 < e, p2 = k + 2 < e;
        const double a0 = p0 ? ldv(v + sc[k]) : 0.0, a1 = p1 ? ldv(v + sc[k + 1]) : 0.0,
                     a2 = p2 ? ldv(v + sc[k + 2]) : 0.0;
        if (p0)
            s += sv[k] * a0;
        if (p1)
            s += sv[k + 1] * a1;
        if (p2)
            s += sv[k + 2] * a2;
        return s;
    };
    auto col_dot = [&](int j, const double *v, bool shared) { return dot(tv, tci, trp[j], trp[j + 1], v, shared); };
    auto row_dot_ = [&](int i, const double *v, bool shared) { return dot(av, aci, arp[i], arp[i + 1], v, shared); };
    const bool hasq = D.q != nullptr;
    ResidentState s = *D.state;
    s.optimal = s.restarts = s.evaluations = 0;
    const int k_begin = s.k;
    double dist_x = 0.0, dist_y = 0.0;
    bool do_restart = false;
    grid_begin(S);
    grid_barrier(S); // every block has read the state and its vectors

    // compute_residual of the stored iterates (residual_kernel and
    // read_residual for a problem without cones)
    auto evaluate = [&](bool want_dist) {
        const double tau = P.step / s.omega;
        const bool l2 = P.l2 != 0;
        auto term = [&](double v) { return l2 ? v * v : abs_or_inf(v); };
        auto acc = [&](double a, double t) { return l2 ? a + t : fmax(a, t); };
        double pr = 0, dr = 0, qn = 0, an = 0, ps = 0, cx = 0, xqx = 0, sx = 0, dx2 = 0, dy2 = 0;
        for (int i = tid; i < nr; i += RT) {
            const double v = row_dot_(i, D.xp, false) + gg[i];
            const double proj = clampd(lc[i], v, uc[i]);
            pr = acc(pr, term((v - proj) * D.cr[w0 + i]));
            const double yv = D.yp[w0 + i];
            const double lf = isfinite(lc[i]) ? lc[i] : 0.0, uf = isfinite(uc[i]) ? uc[i] : 0.0;
            ps += fmax(yv, 0.0) * lf + fmin(yv, 0.0) * uf - gg[i] * yv;
            if (want_dist)
                dy2 += (yv - y0[i]) * (yv - y0[i]);
        }
        for (int j = tid; j < nv; j += RT) {
            const double aty = col_dot(j, D.yp, false), xv = D.xp[c0 + j], vr = D.vr[c0 + j];
            const double qx = q[j] * xv;
            double d, sl;
            if (!hasq) {
                sl = D.ds[c0 + j];
                d = (c[j] - aty - sl) * vr;
            } else {
                const double gr = qx + c[j] - aty, t = xv - tau * gr;
                const double pt = fmax(lo[j], fmin(hi[j], t));
                sl = (pt - t) / tau;
                d = (gr - sl) * vr;
            }
            dr = acc(dr, term(d));
            cx += c[j] * xv;
            xqx += xv * qx;
            sx += sl * xv;
            qn = acc(qn, term(qx * vr));
            an = acc(an, term(aty * vr));
            if (want_dist)
                dx2 += (xv - x0[j]) * (xv - x0[j]);
        }
        double v[RESIDENT_SLOTS] = {pr, dr, qn, an, ps, cx, xqx, sx, dx2, dy2};
        grid_fold<RESIDENT_SLOTS, RWARPS>(v, l2 ? 0u : 0xfu, S, sh);
        auto nrm = [&](double a) { return l2 ? sqrt(a) : a; };
        s.abs_p = nrm(v[0]) / P.sb;
        s.abs_d = nrm(v[1]) / P.sc;
        const double half = hasq ? 0.5 * v[6] : 0.0;
        s.pobj = (v[5] + half) / (P.sb * P.sc) + P.obj_const;
        s.dobj = (v[7] + v[4] - half) / (P.sb * P.sc) + P.obj_const;
        s.rel_p = s.abs_p / (1.0 + P.bnorm);
        const double den = hasq ? 1.0 + fmax(P.cnorm, fmax(nrm(v[2]) / P.sc, nrm(v[3]) / P.sc)) : 1.0 + P.cnorm;
        s.rel_d = s.abs_d / den;
        s.gap = fabs(s.pobj - s.dobj);
        s.rel_gap = s.gap / (1.0 + fabs(s.pobj) + fabs(s.dobj));
        dist_x = sqrt(v[8]);
        dist_y = sqrt(v[9]);
        ++s.evaluations;
    };

    while (s.k < P.iteration_limit) {
        if (s.major || s.k == 0 || s.k % resident_print_frequency(s.k) == 0) {
            // an evaluation of the host's, or the budget is spent
            if ((s.major && s.k < 3 * P.freq) || s.k - k_begin >= P.budget)
                break;
            evaluate(s.major || s.k == 0);
            if (s.rel_d < P.eps_feas && s.rel_p < P.eps_feas && s.rel_gap < P.eps_opt) {
                s.optimal = 1;
                break;
            }
        }
        if (s.major || s.k == 0) {
            do_restart = false;
            if (s.k == P.freq)
                do_restart = true;
            else if (s.k > P.freq) {
                if (s.fpe <= P.sufficient * s.fpe0)
                    do_restart = true;
                if (s.fpe <= P.necessary * s.fpe0 && s.fpe > s.fpe_last)
                    do_restart = true;
                if (s.inner >= P.artificial * s.k)
                    do_restart = true;
            }
            s.fpe_last = s.fpe;
            if (do_restart) {
                const double ratio = s.rel_d / s.rel_p;
                if (dist_x > 1e-16 && dist_y > 1e-16 && dist_x < 1e12 && dist_y < 1e12 && ratio > 1e-8 && ratio < 1e8) {
                    const double err = log(dist_y) - log(dist_x) - log(s.omega);
                    s.err_sum *= P.i_smooth;
                    s.err_sum += err;
                    const double derr = err - s.last_err;
                    s.omega *= exp(P.k_p * err + P.k_i * s.err_sum + P.k_d * derr);
                    s.last_err = err;
                } else {
                    s.omega = s.best_omega;
                    s.err_sum = 0.0;
                    s.last_err = 0.0;
                }
                const double g = fabs(log10(s.rel_d / s.rel_p));
                if (g < s.best_gap) {
                    s.best_gap = g;
                    s.best_omega = s.omega;
                }
                for (int j = tid; j < nv; j += RT)
                    x0[j] = x[j] = D.xp[c0 + j];
                for (int i = tid; i < nr; i += RT) {
                    y0[i] = y[i] = D.yp[w0 + i];
                    __stcg(D.y + w0 + i, y[i]);
                }
                grid_barrier(S);
                ++s.restarts;
                s.inner = 0;
                s.fpe_last = INFINITY;
            }
        }
        s.major = ((s.k + 1) % P.freq) == 0;
        const bool store = s.major || ((s.k + 2) % resident_print_frequency(s.k + 2)) == 0;
        const bool want_fpe = s.major || do_restart;
        const double w = (double)(s.inner + 1) / (s.inner + 2);
        double tau = P.step / s.omega;
        if (P.nonconvexity < 0) {
            tau = fmax(tau, -1.01 * fmin(0.0, P.nonconvexity));
            tau /= 100;
        }
        const double sigma = P.step * s.omega;
        for (int j = tid; j < nv; j += RT) {
            const double xi = x[j], aty = ONE ? col_dot(j, y, true) : col_dot(j, D.y, false);
            double t = xi - tau * (c[j] - aty);
            if (hasq)
                t /= (1.0 + tau * q[j]);
            const double pt = clampd(lo[j], t, hi[j]);
            const double xr = 2.0 * pt - xi;
            if (ONE)
                xrs[j] = xr;
            else
                __stcg(D.xr + c0 + j, xr);
            if (store) {
                D.xp[c0 + j] = pt;
                if (!hasq)
                    D.ds[c0 + j] = (pt - t) / tau;
            }
            if (want_fpe)
                D.dx[c0 + j] = xr - xi;
            const double refl = P.rho * xr + (1.0 - P.rho) * xi;
            x[j] = w * refl + (1.0 - w) * x0[j];
        }
        grid_barrier(S);
        for (int i = tid; i < nr; i += RT) {
            const double yi = y[i];
            const double v = (ONE ? row_dot_(i, xrs, true) : row_dot_(i, D.xr, false)) + gg[i];
            const double pr = clampd(lc[i], v - yi / sigma, uc[i]);
            const double yn = yi - sigma * v + sigma * pr;
            if (store)
                D.yp[w0 + i] = yn;
            const double yr = 2.0 * yn - yi;
            if (want_fpe)
                D.dy[w0 + i] = yr - yi;
            const double refl = P.rho * yr + (1.0 - P.rho) * yi;
            y[i] = w * refl + (1.0 - w) * y0[i];
            if (!ONE)
                __stcg(D.y + w0 + i, y[i]);
        }
        grid_barrier(S);
        if (want_fpe) { // compute_fixed_point_error
            double v[3] = {0.0, 0.0, 0.0};
            for (int j = tid; j < nv; j += RT) {
                const double d = D.dx[c0 + j];
                v[0] += d * d;
                v[2] += col_dot(j, D.dy, false) * d;
            }
            for (int i = tid; i < nr; i += RT) {
                const double d = D.dy[w0 + i];
                v[1] += d * d;
            }
            grid_fold<3, RWARPS>(v, 0u, S, sh);
            s.fpe = sqrt(v[0] * s.omega + v[1] / s.omega + 2 * P.step * v[2]);
            if (do_restart)
                s.fpe0 = s.fpe;
            do_restart = false;
        }
        ++s.inner;
        ++s.k;
    }
    for (int j = tid; j < nv; j += RT) {
        D.x[c0 + j] = x[j];
        D.x0[c0 + j] = x0[j];
        if (ONE)
            D.xr[c0 + j] = xrs[j];
    }
    for (int i = tid; i < nr; i += RT) {
        D.y[w0 + i] = y[i];
        D.y0[w0 + i] = y0[i];
    }
    grid_end(S);
    if (blockIdx.x == 0 && tid == 0) {
        s.wait_failed = gridDim.x > 1 ? *(volatile int *)S.err : 0;
        *D.state = s;
    }
}

static size_t resident_smem(const ResidentPlan &p)
{
    return 8 * ((size_t)p.cap_a + p.cap_at + 6 * (size_t)p.vars + 5 * (size_t)p.rows + (p.blocks == 1 ? p.vars : 0)) +
           4 * ((size_t)p.vars + p.rows + 2 + p.cap_a + p.cap_at);
}

constexpr size_t RESIDENT_SMEM = 216 * 1024;

// Most entries of a block's rows of M when its rows are dealt to `blocks` (by
// count, as the kernel deals them).
__device__ int most_entries(const int *rp, int rows, int blocks)
{
    int most = 0;
    for (int b = threadIdx.x; b < blocks; b += blockDim.x)
        most = max(most, rp[(long long)rows * (b + 1) / blocks] - rp[(long long)rows * b / blocks]);
    return most;
}

// out[0..3]: A's and A^T's most entries of a block at b0 blocks, then at b1
__global__ void resident_share_kernel(int n, int m, const int *A_rp, const int *At_rp, int b0, int b1, int *out)
{
    __shared__ int most[4];
    if (threadIdx.x < 4)
        most[threadIdx.x] = 0;
    __syncthreads();
    atomicMax(&most[0], most_entries(A_rp, m, b0));
    atomicMax(&most[1], most_entries(At_rp, n, b0));
    atomicMax(&most[2], most_entries(A_rp, m, b1));
    atomicMax(&most[3], most_entries(At_rp, n, b1));
    __syncthreads();
    if (threadIdx.x < 4)
        out[threadIdx.x] = most[threadIdx.x];
}

// One block when everything fits in it with at most RESIDENT_ONE variables or
// rows (measured against a grid: one block's barrier is 50 cycles, the grid's
// 1700, and a block's FP64 units take 4 cycles per variable); otherwise about
// a thread per variable, at most one block per SM.  Every block stages its
// rows of A and A^T, so the fullest block decides whether the problem fits: a
// block that reads a matrix from L2 instead, a row per thread, is waited for
// by all others at both barriers (columns of 64 entries side by side in
// 150000 variables: 102 us per iteration, 37 by the kernels of one launch per
// step; 60 entries in 100000: 50 against 35).
constexpr int RESIDENT_ONE = 2048;

// shares: 4 ints of device scratch
ResidentPlan resident_plan(int n, int m, long long nnz, const int *A_rp, const int *At_rp, int sms, int *shares,
                           cudaStream_t s)
{
    auto plan = [&](int blocks, long long a, long long at) {
        ResidentPlan p{};
        p.blocks = blocks;
        p.vars = (n + blocks - 1) / blocks;
        p.rows = (m + blocks - 1) / blocks;
        p.cap_a = (int)a;
        p.cap_at = (int)at;
        p.smem = resident_smem(p);
        return p;
    };
    auto fits = [](const ResidentPlan &p) { return p.smem <= RESIDENT_SMEM && p.vars <= 2 * RT && p.rows <= 2 * RT; };
    if (nnz > (1 << 24))
        return ResidentPlan{};
    ResidentPlan p{};
    if (std::max(n, m) <= RESIDENT_ONE)
        p = plan(1, nnz, nnz);
    if (p.blocks == 0 || p.smem > RESIDENT_SMEM) {
        const long long mean = (nnz + sms - 1) / sms;
        if (!fits(plan(sms, mean, mean)))
            return ResidentPlan{};
        int blocks = std::min(sms, std::max(2, (std::max(n, m) + RT - 1) / RT * 2));
        // with so many entries that a quarter over the mean would not fit, a
        // block per SM: their gathers are what an iteration waits for (rows of
        // 60 entries, 5000 variables: 19.0 us on 20 blocks, 12.1 on 148)
        const long long quarter = (nnz + blocks - 1) / blocks * 5 / 4 + 64;
        if (!fits(plan(blocks, quarter, quarter)))
            blocks = sms;
        int h[4];
        resident_share_kernel<<<1, TPB, 0, s>>>(n, m, A_rp, At_rp, blocks, sms, shares);
        CK(cudaMemcpyAsync(h, shares, sizeof(h), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        p = plan(blocks, h[0], h[1]);
        if (!fits(p))
            p = plan(sms, h[2], h[3]);
        if (!fits(p))
            return ResidentPlan{};
    }
    const void *f = p.blocks == 1 ? (const void *)resident_kernel<true> : (const void *)resident_kernel<false>;
    allow_shared(f, RESIDENT_SMEM);
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, RT, p.smem));
    return per_sm >= 1 ? p : ResidentPlan{};
}

void launch_resident(const ResidentPlan &p, const ResidentData &D, const ResidentParams &P, const GridSlots &S,
                     cudaStream_t s)
{
    void *args[] = {(void *)&D, (void *)&P, (void *)&S, (void *)&p};
    const void *f = p.blocks == 1 ? (const void *)resident_kernel<true> : (const void *)resident_kernel<false>;
    CK(cudaLaunchCooperativeKernel(f, p.blocks, RT, args, p.smem, s));
}

} // namespace pdhcg
