// inner_small.cu -- the inner BB solve (bb.cuh) of problems without cones
// whose quadratic term is a sparse Q with short rows: a latency-bound loop
// (56 inner iterations per outer one on a Q of 1e4 rows and 4e4 entries, all
// of it in L2).
//
// bb_kernel spends 8 us per inner iteration on such a problem (here 4.1): two
// grid.sync over 592 blocks, two folds of 592 partials by every block, and
// the vectors of the iteration reloaded from L2 in every phase.  Here a
// thread owns V variables for the whole solve and keeps everything of them
// in registers (c - A^T y, x, the bounds, the preconditioner, the gradient,
// the iterate and the step), the block's rows of Q lie in shared memory, only
// x_p goes through L2 (its neighbours gather it), and an inner iteration is one
// barrier and one fold over at most one block per SM.
//
// Two forms.  The cluster form runs on one cluster of 16 blocks, whose
// hardware barrier takes 0.25 us where a barrier over the grid takes 1.25, and
// exchanges its sums through distributed shared memory; but 16 SMs gather only
// 0.7 entries of x_p a cycle each, so it is for Q with few entries off the
// diagonal (SMALL_CLUSTER_NNZ).  The grid form takes up to one block per SM.
#include <cooperative_groups.h>

#include "gridsum.cuh"
#include "launch.cuh"

namespace pdhcg {

constexpr int SMALL_CLUSTER = 16;
// Entries of Q off the diagonal up to which the cluster form is taken.  A solve
// of 200 outer iterations with 5 inner ones each, cluster against grid form: 6.2
// / 8.0 ms at 4 K entries (2000 variables), 8.4 / 9.5 at 48 K and 9.7 / 10.3 at
// 80 K (8000), 8.4 / 8.6 at 64 K and 10.0 / 9.5 at 96 K (16000), 21.2 / 11.2 at
// 224 K.
constexpr int SMALL_CLUSTER_NNZ = 64 * 1024;

namespace cgc = cooperative_groups;

// Gathers of one row in flight: ROW_WIDTH, and as many again where one of the
// thread's rows is longer.  An inner iteration waits for its longest row's rounds,
// but every gather that a round has room for costs its issue slots in the short
// rows too.  Us per inner iteration at a fixed 8 / 12 / 16, and with 8 (one row a
// thread) or 6 (two) doubled where needed: Q = B'B with rows to about 20 entries,
// 1000 variables 6.5 / 4.1 / - and 3.9, 10000 7.6 / 5.2 / 5.8 and 5.0;
// tridiagonal, 2000 4.5 / 4.5 / 5.0 and 4.5, 16000 5.3 / 5.5 / 6.1 and 5.1.
template <int V>
constexpr int ROW_WIDTH = V == 1 ? 8 : 6;

// Barriers and sums of the two forms.  fold: both values summed over the
// launch's blocks, in block order, the same in every thread; also a barrier.
// barrier: what any thread wrote to global memory is visible after it.
template <int NT, bool CLUSTER>
struct SmallSync {
    GridSlots &S;
    double *sh;                       // 2 NT / 32 doubles, then grid_fold's
    double (*ex)[2][SMALL_CLUSTER];   // cluster: [parity][value][block]
    int parity = 0;
    __device__ SmallSync(GridSlots &S_, double *sh_, double (*ex_)[2][SMALL_CLUSTER]) : S(S_), sh(sh_), ex(ex_) {}

    __device__ __forceinline__ static void cluster_sync()
    {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    __device__ __forceinline__ void barrier()
    {
        if (CLUSTER)
            cluster_sync();
        else
            grid_barrier(S);
    }
    __device__ __forceinline__ void fold(double &a, double &b)
    {
        if (!CLUSTER) {
            double v[2] = {a, b};
            grid_fold<2, NT / 32>(v, 0u, S, sh);
            a = v[0];
            b = v[1];
            return;
        }
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        a = warp_sum(a);
        b = warp_sum(b);
        if (lane == 0) {
            sh[warp] = a;
            sh[NT / 32 + warp] = b;
        }
        __syncthreads();
        if (warp == 0) { // the block's sums into every block's row
            a = warp_sum(lane < NT / 32 ? sh[lane] : 0.0);
            b = warp_sum(lane < NT / 32 ? sh[NT / 32 + lane] : 0.0);
            cgc::cluster_group cl = cgc::this_cluster();
            const int me = (int)cl.block_rank();
            if (lane < SMALL_CLUSTER) {
                double *row = cl.map_shared_rank(&ex[parity][0][0], lane);
                row[me] = a;
                row[SMALL_CLUSTER + me] = b;
            }
        }
        cluster_sync();
        // lanes 0-15 add the first value, 16-31 the second, then exchange
        double v = ex[parity][lane >> 4][lane & 15];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
            v += __shfl_xor_sync(FULL, v, o);
        a = __shfl_sync(FULL, v, 0);
        b = __shfl_sync(FULL, v, 16);
        parity ^= 1;
    }
};

template <int NT, int V, bool CLUSTER>
__global__ void __launch_bounds__(NT) bb_small_kernel(BBData D, BBParams P, GridSlots S, int cap)
{
    extern __shared__ __align__(16) char sm[];
    __shared__ double sh[2 * (NT / 32 + 1)];
    __shared__ double ex[2][2][SMALL_CLUSTER];
    static_assert(NT >= 64, "grid_fold takes a warp per value");
    SmallSync<NT, CLUSTER> sync(S, sh, ex);
    double *sv = (double *)sm;
    int *sc = (int *)(sm + sizeof(double) * cap);
    const int nb = gridDim.x, tid = threadIdx.x;
    const int r0 = (int)((long long)D.n * blockIdx.x / nb), r1 = (int)((long long)D.n * (blockIdx.x + 1) / nb);
    const int q0 = D.Q_rp[r0], q1 = D.Q_rp[r1];
    for (int e = tid; e < q1 - q0; e += NT) {
        sc[e] = D.Q_ci[q0 + e];
        sv[e] = D.Q_vf ? (double)D.Q_vf[q0 + e] : D.Q_v[q0 + e];
    }
    if (!CLUSTER)
        grid_begin(S);
    const double inv_tau = 1.0 / P.tau;
    double alpha0 = 1.0 / inv_tau;
    if (D.m_inv) {
        const double ts = *D.tol_scale;
        alpha0 *= ts * ts;
    }
    const double tol = *D.tol;
    int b[V], e[V];
    double cb[V], x[V], lo[V], hi[V], mi[V], md[V], dq[V], g[V], xp[V], dir[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int j = r0 + tid + NT * v;
        const bool ok = j < r1;
        b[v] = ok ? D.Q_rp[j] - q0 : 0;
        e[v] = ok ? D.Q_rp[j + 1] - q0 : 0;
        cb[v] = ok ? D.c[j] - D.aty[j] : 0.0;
        x[v] = ok ? D.x[j] : 0.0;
        lo[v] = ok ? D.l[j] : 0.0;
        hi[v] = ok ? D.u[j] : 0.0;
        mi[v] = ok && D.m_inv ? D.m_inv[j] : 1.0;
        md[v] = ok && D.m_diag ? D.m_diag[j] : 1.0;
        dq[v] = 0.0;
    }
    __syncthreads();
    // the diagonal entries, whose operand the thread holds, leave the staged
    // rows (the later entries move up)
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int j = r0 + tid + NT * v;
        int w = b[v];
        for (int k = b[v]; k < e[v]; ++k) {
            if (sc[k] == j) {
                dq[v] += sv[k];
            } else {
                sc[w] = sc[k];
                sv[w] = sv[k];
                ++w;
            }
        }
        e[v] = w;
    }
    // s = (Q w) of the thread's rows (the diagonal's operands are `own`), the rows
    // side by side with up to 2 ROW_W gathers of each in flight, entries in order
    int longest = 0;
#pragma unroll
    for (int v = 0; v < V; ++v)
        longest = max(longest, e[v] - b[v]);
    constexpr int ROW_W = ROW_WIDTH<V>;
    auto rows = [&](const double *w, const double (&own)[V], double (&s)[V]) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            s[v] = dq[v] * own[v];
#pragma unroll 1
        for (int k = 0; k < longest; k += 2 * ROW_W) {
            const bool more = longest > k + ROW_W;
            double a[V][2 * ROW_W];
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int u = 0; u < ROW_W; ++u)
                    a[v][u] = b[v] + k + u < e[v] ? __ldcg(w + sc[b[v] + k + u]) : 0.0;
            if (more)
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int u = ROW_W; u < 2 * ROW_W; ++u)
                        a[v][u] = b[v] + k + u < e[v] ? __ldcg(w + sc[b[v] + k + u]) : 0.0;
#pragma unroll
            for (int v = 0; v < V; ++v)
#pragma unroll
                for (int u = 0; u < ROW_W; ++u)
                    if (b[v] + k + u < e[v])
                        s[v] += sv[b[v] + k + u] * a[v][u];
            if (more)
#pragma unroll
                for (int v = 0; v < V; ++v)
#pragma unroll
                    for (int u = ROW_W; u < 2 * ROW_W; ++u)
                        if (b[v] + k + u < e[v])
                            s[v] += sv[b[v] + k + u] * a[v][u];
        }
    };
    // the projected step from `from` along M^-1 g; the partial of dir' M dir
    auto var_step = [&](double alpha, const double (&from)[V]) {
        double part = 0.0;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int j = r0 + tid + NT * v;
            if (j < r1) {
                const double xn = clampd(lo[v], from[v] - alpha * mi[v] * g[v], hi[v]);
                dir[v] = xn - from[v];
                xp[v] = xn;
                __stcg(D.xp + j, xn);
                part += dir[v] * md[v] * dir[v];
            }
        }
        return part;
    };
    double qv[V];
    rows(D.x, x, qv);
#pragma unroll
    for (int v = 0; v < V; ++v) {
        dir[v] = xp[v] = 0.0;
        g[v] = qv[v] + cb[v];
    }
    // A step's dir' M dir is wanted for the convergence test and the next step
    // length, both after the gradient at x_p is there; so the step only passes
    // a barrier (x_p must be visible) and its sum rides along with the
    // gradient's (the gradient after the last step is formed in vain).
    double ss = var_step(alpha0, x);
    sync.barrier();
    int it = 1;
    for (;;) {
        double t = 0.0;
        if (it < D.limit) {
            rows(D.xp, xp, qv);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const double gn = qv[v] + cb[v] + inv_tau * (xp[v] - x[v]);
                t += dir[v] * (gn - g[v]);
                g[v] = gn;
            }
        }
        sync.fold(ss, t);
        if (it >= D.limit || sqrt(ss) <= tol)
            break;
        ss = var_step(ss / t, xp);
        sync.barrier();
        ++it;
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const int j = r0 + tid + NT * v;
        if (j < r1) {
            const double xr = 2.0 * xp[v] - x[v];
            D.xr[j] = xr;
            if (P.want_fpe)
                D.dx[j] = xr - x[v];
            const double refl = P.rho * xr + (1.0 - P.rho) * x[v];
            D.x[j] = P.w * refl + (1.0 - P.w) * D.x0[j];
        }
    }
    if (!CLUSTER)
        grid_end(S);
    if (blockIdx.x == 0 && tid == 0)
        *D.inner_total += it - 1;
}

// Launch shapes.  Cluster: 16 blocks, the fewest threads that hold the
// variables.  Grid: the smallest blocks that fit one per SM (a smaller block
// reduces and synchronises faster).  cap: entries of Q that a block has room
// for at least (the fullest block may raise it).
struct SmallShape {
    const void *kernel;
    int threads, vars, cap;
};

static SmallShape cluster_shape(int n)
{
    if (n <= SMALL_CLUSTER * 128)
        return {(const void *)bb_small_kernel<128, 1, true>, 128, 128, 8192};
    if (n <= SMALL_CLUSTER * 512)
        return {(const void *)bb_small_kernel<512, 1, true>, 512, 512, 8192};
    if (n <= SMALL_CLUSTER * 1024)
        return {(const void *)bb_small_kernel<512, 2, true>, 512, 1024, 8192};
    return {nullptr, 0, 0, 0};
}

static SmallShape grid_shape(int n, int sms)
{
    if (n <= sms * 128)
        return {(const void *)bb_small_kernel<128, 1, false>, 128, 128, 2048};
    if (n <= sms * 256)
        return {(const void *)bb_small_kernel<256, 1, false>, 256, 256, 4096};
    if (n <= sms * 512)
        return {(const void *)bb_small_kernel<512, 1, false>, 512, 512, 8192};
    if (n <= sms * 1024)
        return {(const void *)bb_small_kernel<512, 2, false>, 512, 1024, 16384};
    return {nullptr, 0, 0, 0};
}

static cudaLaunchConfig_t small_config(const SmallPlan &p, cudaLaunchAttribute *at, cudaStream_t s)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(p.blocks);
    c.blockDim = dim3(p.threads);
    c.dynamicSmemBytes = (size_t)p.cap * 12;
    c.stream = s;
    if (p.cluster) {
        at->id = cudaLaunchAttributeClusterDimension;
        at->val.clusterDim.x = SMALL_CLUSTER;
        at->val.clusterDim.y = at->val.clusterDim.z = 1;
    } else {
        at->id = cudaLaunchAttributeCooperative;
        at->val.cooperative = 1;
    }
    c.attrs = at;
    c.numAttrs = 1;
    return c;
}

// most entries of a block's rows at b0 and at b1 blocks (rows dealt by count)
__global__ void small_share_kernel(int n, const int *rp, int b0, int b1, int *out)
{
    __shared__ int most[2];
    if (threadIdx.x < 2)
        most[threadIdx.x] = 0;
    __syncthreads();
    for (int which = 0; which < 2; ++which) {
        const int nb = which ? b1 : b0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x)
            atomicMax(&most[which], rp[(long long)n * (b + 1) / nb] - rp[(long long)n * b / nb]);
    }
    __syncthreads();
    if (threadIdx.x < 2)
        out[threadIdx.x] = most[threadIdx.x];
}

constexpr int SMALL_CAP = 200 * 1024 / 12; // entries of Q that a block can stage

// The shape for an n x n Q, blocks = 0: none.  Every block stages its rows, so
// a shape is taken only if its fullest block fits: rows read from L2 by a
// thread each are what all blocks then wait for (500 rows of 60 entries side
// by side in 10000: 240 us per outer iteration that way, 113 by the general
// kernel; 3000 in 60000: 384 against 201).  shares: 2 ints of device scratch.
SmallPlan bb_small_plan(int n, long long nnz, const int *Q_rp, int sms, int *shares, cudaStream_t s)
{
    // (every row of Q has a diagonal entry in practice)
    const SmallShape cl = nnz - n <= SMALL_CLUSTER_NNZ ? cluster_shape(n) : SmallShape{}, gr = grid_shape(n, sms);
    if (!cl.kernel && !gr.kernel)
        return SmallPlan{};
    const int grid = gr.kernel ? std::max((n + gr.vars - 1) / gr.vars, 1) : 1;
    int h[2];
    small_share_kernel<<<1, TPB, 0, s>>>(n, Q_rp, SMALL_CLUSTER, grid, shares);
    CK(cudaMemcpyAsync(h, shares, sizeof(h), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (cl.kernel && h[0] <= SMALL_CAP) {
        const SmallPlan p{cl.kernel, SMALL_CLUSTER, cl.threads, std::max(cl.cap, h[0]), true};
        allow_shared(p.kernel, (size_t)SMALL_CAP * 12);
        CK(cudaFuncSetAttribute(p.kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        cudaLaunchAttribute at;
        const cudaLaunchConfig_t c = small_config(p, &at, nullptr);
        int clusters = 0;
        CK(cudaOccupancyMaxActiveClusters(&clusters, p.kernel, &c));
        if (clusters >= 1)
            return p;
    }
    if (gr.kernel && h[1] <= SMALL_CAP) {
        const SmallPlan p{gr.kernel, grid, gr.threads, std::max(gr.cap, h[1]), false};
        allow_shared(p.kernel, (size_t)SMALL_CAP * 12);
        int per_sm = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, p.threads, (size_t)p.cap * 12));
        if (per_sm >= 1 && grid <= sms)
            return p;
    }
    return SmallPlan{};
}

void launch_bb_small(const SmallPlan &p, const BBData &D, const BBParams &P, const GridSlots &S, cudaStream_t s)
{
    cudaLaunchAttribute at;
    const cudaLaunchConfig_t c = small_config(p, &at, s);
    void *args[] = {(void *)&D, (void *)&P, (void *)&S, (void *)&p.cap};
    CK(cudaLaunchKernelExC(&c, p.kernel, args));
}

} // namespace pdhcg
