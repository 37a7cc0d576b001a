// inner_dense.cu -- the inner BB solve (bb.cuh) when the quadratic term is a
// dense low-rank R^T D R over the leading w columns plus at most a diagonal
// Q (the portfolio objective): one pass over R per inner iteration.
//
// What bounds it: R is k x w doubles (160 MB at k = 100, w = 2e5) and is read
// from HBM in every pass.  bb_kernel takes two passes per inner iteration,
// R^T (D R x_p) for the gradient and, after the step, R x_p for the next one,
// because the BB step length needs dir . (g_new - g) before it can step, and
// that takes the first pass.  But g_new - g = H dir, so
//   dir . (g_new - g) = dir . (Q + I / tau) dir + (R dir)^T D (R dir),
// and R dir is what a pass can add up anyway while a column of R is at hand:
// a pass takes a tile of columns, forms their gradient from D R x_p, steps,
// and adds R dir of the tile.  The sums of a pass (dir' M dir, dir . (Q + I /
// tau) dir, and the k-vector R dir) give the next step length and, by
// R x_p += R dir, the next gradient, so R is read once, and one grid barrier
// ends a pass instead of four.  R x at the start of a solve follows from the
// last one by the same linear combination as x itself (reflection and
// Halpern average); it is formed anew by a pass of its own at every restart
// (BBParams.refresh), so rounding does not build up.
//
// R is laid out once per solve in tiles of 32 columns, k x 32 values back to
// back, so a tile is one contiguous bulk copy into shared memory (TMA,
// cp.async.bulk) that completes on an mbarrier; as many tiles are in flight
// as shared memory holds.  Passes alternate their direction over a block's
// tiles: the last ones read are the first ones of the next pass and come from
// L2.  Warps 0-15 multiply (warp i the rows i, i + 16, ...; a lane per
// column), U warps step a tile's 32 variables each, one issues the copies,
// one takes the variables and cone blocks past w, which R does not touch.
// The step of a tile is a chain (the row sums from shared memory, the
// variables' data from L2, a dozen dependent FP64 operations, two block
// barriers) of about 1 us, more than the tile's share of HBM time, so U tiles
// go through it side by side: 4, 2 or 1, as many as shared memory holds twice
// with enough copies in flight behind them (dense_form).
#include "gridsum.cuh"
#include "launch.cuh"

namespace pdhcg {

constexpr int DT = 32;                   // columns of a tile
constexpr int DW = 16;                   // multiplying warps
constexpr int DENSE_MAX_STAGES = 24;
constexpr int DENSE_AHEAD = 8; // tiles between the L2 prefetch of a tile's vectors and their use
constexpr int dense_threads(int u) { return 32 * (DW + u + 2); }

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *b, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(unsigned long long *b)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(smem_addr(b)) : "memory");
}

__device__ __forceinline__ void mbar_expect(unsigned long long *b, unsigned bytes)
{
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n\t}" ::"r"(smem_addr(b)),
                 "r"(bytes)
                 : "memory");
}

// waits for the phase with this parity to complete; false when SPIN_LIMIT ran out
__device__ __forceinline__ bool mbar_wait(unsigned long long *b, unsigned parity, int *err)
{
    for (int spin = 0; spin < SPIN_LIMIT; ++spin) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(smem_addr(b)), "r"(parity)
                     : "memory");
        if (done)
            return true;
        if ((spin & 1023) == 1023 && *(volatile int *)err)
            break;
    }
    *err = 1;
    return false;
}

__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, unsigned long long *b)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(b))
                 : "memory");
}

// One cone block past w: candidate from the gradient without R, projection,
// the block's parts of dir' M dir and dir . (Q + I / tau) dir.
template <int S>
__device__ __forceinline__ void dense_cone_block(const BBData &D, const DenseR &R, bool init, double alpha,
                                                 double inv_tau, int cb, int lane, double &sms, double &sqs)
{
    const int st = D.cone_start[cb], L = D.cone_len[cb], type = D.cone_type[cb];
    WarpSlots<S> sl;
    double xo[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        sl.x[s] = 0.0;
        sl.d[s] = sl.w[s] = 1.0;
        xo[s] = 0.0;
        if (i < L) {
            const int j = st + i;
            xo[s] = init ? D.x[j] : D.xp[j];
            double g = (R.qd ? R.qd[j] * xo[s] : 0.0) + D.c[j] - D.aty[j];
            if (!init)
                g += inv_tau * (xo[s] - D.x[j]);
            sl.x[s] = clampd(D.l[j], xo[s] - alpha * (D.m_inv ? D.m_inv[j] : 1.0) * g, D.u[j]);
            sl.d[s] = D.vr[j];
        }
    }
    const bool uni = warp_uniform_unit<S>(sl, L, lane);
    warp_project<S, CONES_WIDE | CONES_THREE>(type, sl, L, lane, uni, D.cone_warm ? D.cone_warm + cb : nullptr,
                                              D.cone_alpha ? D.cone_alpha[cb] : 0.0);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        if (i < L) {
            const int j = st + i;
            const double d = sl.x[s] - xo[s];
            D.xp[j] = sl.x[s];
            sms += d * (D.m_diag ? D.m_diag[j] : 1.0) * d;
            sqs += d * ((R.qd ? R.qd[j] : 0.0) + inv_tau) * d;
        }
    }
}

// x_refl, dx and the Halpern average of one variable
__device__ __forceinline__ void dense_finish(const BBData &D, const BBParams &P, int j, double p)
{
    const double xi = D.x[j], xr = 2.0 * p - xi;
    D.xr[j] = xr;
    if (P.want_fpe)
        D.dx[j] = xr - xi;
    const double refl = P.rho * xr + (1.0 - P.rho) * xi;
    D.x[j] = P.w * refl + (1.0 - P.w) * D.x0[j];
}

// RPW: rows per multiplying warp (k <= DW * RPW); U: tiles of a group
template <typename T, int RPW, int S, int U>
__global__ void __launch_bounds__(32 * (DW + U + 2), 1)
    bb_dense_kernel(BBData D, BBParams P, DenseR R, GridSlots G, int stages)
{
    constexpr int DTHREADS = 32 * (DW + U + 2);
    extern __shared__ __align__(128) char sm[];
    __shared__ unsigned long long full[DENSE_MAX_STAGES], empty[DENSE_MAX_STAGES];
    __shared__ double sstep[2][U][DT];
    __shared__ double drx[DW * RPW], rx[DW * RPW], rs[DW * RPW];
    __shared__ double red[2][U + 1], out[3];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = gridDim.x, k = D.k;
    const int t0 = (int)((long long)R.tiles * blockIdx.x / nb), t1 = (int)((long long)R.tiles * (blockIdx.x + 1) / nb);
    const int nt = t1 - t0;
    const unsigned tile_bytes = (unsigned)(k * DT * sizeof(T));
    const T *tiles = (const T *)R.tile;
    // row sums of a group's tiles by warp, behind the stages
    double (*qpart)[U][DW][DT] = reinterpret_cast<double (*)[U][DW][DT]>(sm + (size_t)stages * tile_bytes);
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], DW);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const double inv_tau = 1.0 / P.tau;
    double alpha0 = 1.0 / inv_tau;
    if (D.m_inv) {
        const double ts = *D.tol_scale;
        alpha0 *= ts * ts;
    }
    const double tol = *D.tol;
    grid_begin(G);
    __syncthreads();

    // A place in the ring of stages: the stage and the parity of its current
    // round, moved on tile by tile.  Readers and the producer each keep their own.
    struct Ring {
        int st = 0;
        unsigned parity = 0;
        __device__ __forceinline__ void next(int stages)
        {
            if (++st == stages) {
                st = 0;
                parity ^= 1u;
            }
        }
    };
    Ring rd, wr; // next tile to read; next stage to fill
    bool wrapped = false; // producer: every stage was filled once
    int pass = 0;
    int pre = 0; // producer: tiles of the next pass already issued
    auto tile_at = [&](int p, int i) { return (p & 1) ? t1 - 1 - i : t0 + i; };
    auto tile_of = [&](int st) { return (const T *)(sm + (size_t)st * tile_bytes); };
    // copies of pass p's tiles [from, to), each once its stage is free
    auto issue = [&](int p, int from, int to) {
        for (int i = from; i < to; ++i) {
            if (wrapped && !mbar_wait(&empty[wr.st], wr.parity ^ 1u, G.err))
                return;
            mbar_expect(&full[wr.st], tile_bytes);
            bulk_load(sm + (size_t)wr.st * tile_bytes, tiles + (size_t)tile_at(p, i) * k * DT, tile_bytes, &full[wr.st]);
            wr.next(stages);
            wrapped = wrapped || wr.st == 0;
        }
    };

    // mode 0: R v alone (v = xv), into rs; 1: first step from x; 2: next step
    // from x_p.  Afterwards rs = R dir (R v) and, for the steps, out[0] =
    // dir' M dir, out[1] = dir . (Q + I / tau) dir over the grid.
    auto run_pass = [&](int mode, double alpha, const double *xv) {
        double sms = 0.0, sqs = 0.0;
        if (warp < DW) {
            double acc[RPW];
#pragma unroll
            for (int a = 0; a < RPW; ++a)
                acc[a] = 0.0;
            double dr[RPW]; // D R x_p of this warp's rows
#pragma unroll
            for (int a = 0; a < RPW; ++a)
                dr[a] = mode && warp + DW * a < k ? drx[warp + DW * a] : 0.0;
            int cur[U], prev[U]; // stages of the group's tiles and of the last group's (a missing one: the first)
            int np = 0;          // tiles of the last group
            for (int i0 = 0; i0 < nt + U; i0 += U) {
                const int nc = max(0, min(U, nt - i0)), b = (i0 / U) & 1;
                if (nc > 0) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        cur[u] = u < nc ? rd.st : cur[0];
                        if (u < nc) {
                            mbar_wait(&full[rd.st], rd.parity, G.err);
                            rd.next(stages);
                        }
                    }
                    if (mode) { // R^T (D R x_p) of the tiles' columns, this warp's rows
                        double q[U];
                        const T *tl[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            q[u] = 0.0;
                            tl[u] = tile_of(cur[u]) + lane;
                        }
#pragma unroll
                        for (int a = 0; a < RPW; ++a) {
                            const int r = warp + DW * a;
                            if (r < k)
#pragma unroll
                                for (int u = 0; u < U; ++u)
                                    q[u] += (double)tl[u][r * DT] * dr[a];
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            qpart[b][u][warp][lane] = q[u];
                    }
                }
                asm volatile("bar.sync 1, %0;" ::"r"(32 * (DW + U)) : "memory");
                if (np > 0) { // R dir of the last group
                    const T *tl[U];
                    double sv[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        tl[u] = tile_of(prev[u]) + lane;
                        sv[u] = u < np ? sstep[b ^ 1][u][lane] : 0.0;
                    }
#pragma unroll
                    for (int a = 0; a < RPW; ++a) {
                        const int r = warp + DW * a;
                        if (r < k)
#pragma unroll
                            for (int u = 0; u < U; ++u)
                                acc[a] += (double)tl[u][r * DT] * sv[u];
                    }
                    __syncwarp();
                    if (lane < np)
                        mbar_arrive(&empty[prev[0] + lane < stages ? prev[0] + lane : prev[0] + lane - stages]);
                }
                np = nc;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    prev[u] = cur[u];
            }
#pragma unroll
            for (int a = 0; a < RPW; ++a) {
                const int r = warp + DW * a;
                const double v = warp_sum(acc[a]);
                if (r < k && lane == 0)
                    __stcg(grid_part(G, 2 + r) + blockIdx.x, v);
            }
        } else if (warp < DW + U) {
            // a tile's 32 variables; their data is loaded a group ahead, and
            // asked into L2 DENSE_AHEAD tiles ahead (R streams through L2 and
            // has evicted it since the last pass)
            const int uw = warp - DW;
            auto ask = [&](const double *v, int j) { asm volatile("prefetch.global.L2 [%0];" ::"l"(v + j)); };
            auto ahead = [&](int i) {
                const int j = tile_at(pass, i) * DT + lane;
                if (i >= nt || j >= R.width || (lane & 3))
                    return; // a lane per 32-byte sector
                if (!mode) {
                    ask(xv, j);
                    return;
                }
                ask(D.x, j);
                if (mode == 2)
                    ask(D.xp, j);
                ask(D.c, j);
                ask(D.aty, j);
                ask(D.l, j);
                ask(D.u, j);
                if (D.m_inv) {
                    ask(D.m_inv, j);
                    ask(D.m_diag, j);
                }
                if (R.qd)
                    ask(R.qd, j);
            };
            double n_xo, n_x, n_c, n_lo, n_hi, n_mi, n_md, n_qd;
            auto fetch = [&](int i) {
                const int j = tile_at(pass, i) * DT + lane;
                const bool ok = i < nt && j < R.width;
                n_xo = n_x = n_c = n_lo = n_hi = n_qd = 0.0;
                n_mi = n_md = 1.0;
                if (!ok)
                    return;
                if (!mode) {
                    n_xo = xv[j];
                    return;
                }
                n_x = D.x[j];
                n_xo = mode == 1 ? n_x : D.xp[j];
                n_c = D.c[j] - D.aty[j];
                n_lo = D.l[j];
                n_hi = D.u[j];
                if (D.m_inv) {
                    n_mi = D.m_inv[j];
                    n_md = D.m_diag[j];
                }
                if (R.qd)
                    n_qd = R.qd[j];
            };
            for (int i = uw + U; i < DENSE_AHEAD; i += U)
                ahead(i);
            fetch(uw);
            for (int i0 = 0; i0 < nt + U; i0 += U) {
                asm volatile("bar.sync 1, %0;" ::"r"(32 * (DW + U)) : "memory");
                const int i = i0 + uw, b = (i0 / U) & 1;
                if (i >= nt)
                    continue;
                ahead(i + DENSE_AHEAD);
                const double xo = n_xo, x = n_x, c = n_c, lo = n_lo, hi = n_hi, mi = n_mi, md = n_md, qd = n_qd;
                const int j = tile_at(pass, i) * DT + lane;
                fetch(i + U);
                if (!mode) {
                    sstep[b][uw][lane] = xo;
                    continue;
                }
                double qw[DW];
#pragma unroll
                for (int w = 0; w < DW; ++w)
                    qw[w] = qpart[b][uw][w][lane];
#pragma unroll
                for (int h = DW / 2; h > 0; h >>= 1)
#pragma unroll
                    for (int w = 0; w < h; ++w)
                        qw[w] += qw[w + h];
                const double q = qd * xo + qw[0];
                double g = q + c;
                if (mode == 2)
                    g += inv_tau * (xo - x);
                double d = 0.0;
                if (j < R.width) {
                    const double xn = clampd(lo, xo - alpha * mi * g, hi);
                    d = xn - xo;
                    D.xp[j] = xn;
                    sms += d * md * d;
                    sqs += d * (qd + inv_tau) * d;
                }
                sstep[b][uw][lane] = d;
            }
            sms = warp_sum(sms);
            sqs = warp_sum(sqs);
            if (lane == 0) {
                red[0][uw] = sms;
                red[1][uw] = sqs;
            }
        } else if (warp == DW + U) {
            if (lane == 0) {
                issue(pass, pre, nt);
                pre = min(nt, stages - 1); // the next pass's first tiles, as the stages come free
                issue(pass + 1, 0, pre);
            }
            __syncwarp();
        } else {
            if (mode) { // variables outside the cones past w, then the cone blocks
                const int nf = D.n_cones > 0 ? D.n_free : D.n;
                for (int r = R.width + 32 * blockIdx.x + lane; r < nf; r += 32 * nb) {
                    const int j = D.free_idx ? D.free_idx[r] : r;
                    const double xo = mode == 1 ? D.x[j] : D.xp[j], qd = R.qd ? R.qd[j] : 0.0;
                    double g = qd * xo + D.c[j] - D.aty[j];
                    if (mode == 2)
                        g += inv_tau * (xo - D.x[j]);
                    const double xn = clampd(D.l[j], xo - alpha * (D.m_inv ? D.m_inv[j] : 1.0) * g, D.u[j]);
                    const double d = xn - xo;
                    D.xp[j] = xn;
                    sms += d * (D.m_diag ? D.m_diag[j] : 1.0) * d;
                    sqs += d * (qd + inv_tau) * d;
                }
                __syncwarp();
                for (int cb = blockIdx.x; cb < D.n_cones; cb += nb) {
                    if (S > 1 && (D.cone_type[cb] == 2 || D.cone_type[cb] == 3))
                        dense_cone_block<1>(D, R, mode == 1, alpha, inv_tau, cb, lane, sms, sqs);
                    else
                        dense_cone_block<S>(D, R, mode == 1, alpha, inv_tau, cb, lane, sms, sqs);
                }
            }
            sms = warp_sum(sms);
            sqs = warp_sum(sqs);
            if (lane == 0) {
                red[0][U] = sms;
                red[1][U] = sqs;
            }
        }
        if (warp >= DW) // the others' place in the ring (only the producer's last wait uses it)
            for (int i = 0; i < nt; ++i)
                rd.next(stages);
        ++pass;
        // the barrier, then the grid's sums: values 0 and 1 are the scalars,
        // 2 + r the rows of R dir
        __syncthreads();
        if (tid == 0) {
            double a = red[0][0], b = red[1][0];
#pragma unroll
            for (int u = 1; u <= U; ++u) {
                a += red[0][u];
                b += red[1][u];
            }
            __stcg(grid_part(G, 0) + blockIdx.x, a);
            __stcg(grid_part(G, 1) + blockIdx.x, b);
            grid_arrive_wait(G);
        }
        __syncthreads();
        constexpr int NW = DTHREADS / 32, F = 4; // rows folded side by side (one after another: 0.5 us each)
        for (int r0 = warp; r0 < k + 2; r0 += NW * F) {
            double a[F] = {};
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int r = r0 + NW * f;
                if (r < k + 2) {
                    const double *p = grid_part(G, r);
#pragma unroll 5
                    for (int b = lane; b < nb; b += 32)
                        a[f] += __ldcg(p + b);
                }
            }
#pragma unroll
            for (int f = 0; f < F; ++f)
                a[f] = warp_sum(a[f]);
#pragma unroll
            for (int f = 0; f < F; ++f) {
                const int r = r0 + NW * f;
                if (lane == 0 && r < k + 2)
                    (r < 2 ? out[r] : rs[r - 2]) = a[f];
            }
        }
        ++G.epoch;
        __syncthreads();
    };
    // D v for the k-vector v, row r
    auto d_row = [&](const double *v, int r) {
        if (D.dkind == 1)
            return D.Ddiag[r] * v[r];
        if (D.dkind == 2) { // symmetric, upper triangle
            double a = 0.0;
            for (int c = 0; c < k; ++c)
                a += D.Ddense[(size_t)min(r, c) * k + max(r, c)] * v[c];
            return a;
        }
        return v[r];
    };
    auto take_rx = [&](const double *xv, double *keep) { // rx = R xv, kept for the next solve
        run_pass(0, 0.0, xv);
        for (int r = tid; r < k; r += DTHREADS) {
            rx[r] = rs[r];
            if (keep && blockIdx.x == 0)
                keep[r] = rs[r];
        }
        __syncthreads();
    };
    double *rx0 = R.rx_state, *rxx = R.rx_state + k; // R x_init and R x
    if (P.refresh == 2)
        take_rx(D.x0, rx0);
    if (P.refresh)
        take_rx(D.x, P.refresh == 1 ? rx0 : nullptr); // 1: x = x_init
    else {
        for (int r = tid; r < k; r += DTHREADS)
            rx[r] = rxx[r];
        __syncthreads();
    }
    // R x of this solve's x stays in registers of the threads that own a row
    double rx_start = tid < k ? rx[tid] : 0.0;
    static_assert(DW * RPW <= DTHREADS, "a thread per row of R");
    for (int r = tid; r < k; r += DTHREADS)
        drx[r] = d_row(rx, r);
    __syncthreads();
    int it = 1;
    for (int mode = 1;; mode = 2) {
        double alpha = alpha0;
        if (mode == 2) {
            if (it >= D.limit || sqrt(out[0]) <= tol)
                break;
            ++it;
            alpha = out[0] / (out[1] + out[2]);
        }
        run_pass(mode, alpha, nullptr);
        // R x_p += R dir, D R x_p, and (R dir)^T D (R dir)
        for (int r = tid; r < k; r += DTHREADS)
            rx[r] += rs[r];
        if (warp == 0) {
            double a = 0.0;
            for (int r = lane; r < k; r += 32)
                a += rs[r] * d_row(rs, r);
            a = warp_sum(a);
            if (lane == 0)
                out[2] = a;
        }
        __syncthreads();
        for (int r = tid; r < k; r += DTHREADS)
            drx[r] = d_row(rx, r);
        __syncthreads();
    }
    // no copy may be in flight when the block's shared memory goes away
    if (warp == DW + U && lane == 0)
        for (int i = 0; i < pre; ++i, rd.next(stages))
            mbar_wait(&full[rd.st], rd.parity, G.err);
    for (int j = t0 * DT + tid; j < min(t1 * DT, R.width); j += DTHREADS)
        dense_finish(D, P, j, D.xp[j]);
    if (warp == DW + U + 1) { // past w: the warp that stepped them
        const int nf = D.n_cones > 0 ? D.n_free : D.n;
        for (int r = R.width + 32 * blockIdx.x + lane; r < nf; r += 32 * nb) {
            const int j = D.free_idx ? D.free_idx[r] : r;
            dense_finish(D, P, j, D.xp[j]);
        }
        for (int cb = blockIdx.x; cb < D.n_cones; cb += nb)
            for (int i = lane; i < D.cone_len[cb]; i += 32)
                dense_finish(D, P, D.cone_start[cb] + i, D.xp[D.cone_start[cb] + i]);
    }
    grid_end(G);
    if (blockIdx.x == 0) {
        if (tid < k) { // R x of the next solve's x
            const double rp = rx[tid], rr = 2.0 * rp - rx_start;
            rxx[tid] = P.w * (P.rho * rr + (1.0 - P.rho) * rx_start) + (1.0 - P.w) * rx0[tid];
        }
        if (tid == 0)
            *D.inner_total += it - 1;
    }
}

// R (row-major, k x width, rows rp[r]) into tiles of DT columns, zero past the width
template <typename T>
__global__ void dense_tile_kernel(int k, int width, const int *rp, const double *v, int tiles, T *tile)
{
    const long long total = (long long)tiles * k * DT;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
         e += (long long)gridDim.x * blockDim.x) {
        const int lane = (int)(e % DT), r = (int)((e / DT) % k), t = (int)(e / ((long long)DT * k));
        const int j = t * DT + lane;
        tile[e] = j < width ? (T)v[(long long)rp[r] + j] : (T)0;
    }
}

// the diagonal of Q, and *bad when it has an entry off the diagonal
__global__ void dense_qdiag_kernel(int n, const int *rp, const int *ci, const double *v, double *qd, int *bad)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int e = rp[i]; e < rp[i + 1]; ++e) {
            if (ci[e] == i)
                s += v[e];
            else
                atomicOr(bad, 1);
        }
        qd[i] = s;
    }
}

void dense_tiles(int k, int width, const int *rp, const double *v, int tiles, double *d, float *f, cudaStream_t s)
{
    const long long total = (long long)tiles * k * DT;
    if (d)
        dense_tile_kernel<double><<<grid_for(total, TPB), TPB, 0, s>>>(k, width, rp, v, tiles, d);
    if (f)
        dense_tile_kernel<float><<<grid_for(total, TPB), TPB, 0, s>>>(k, width, rp, v, tiles, f);
}

void dense_qdiag(int n, const int *rp, const int *ci, const double *v, double *qd, int *bad, cudaStream_t s)
{
    dense_qdiag_kernel<<<grid_for(n, TPB), TPB, 0, s>>>(n, rp, ci, v, qd, bad);
}

int dense_tile_count(int width) { return (width + DT - 1) / DT; }

// Kernel and stages.  Tiles of a group: 4 up to 64 rows, 2 up to 128 where six
// stages fit (FP64: up to 108 rows), else 1, with three stages or more.
struct DenseForm {
    const void *kernel;
    int threads, stages;
    size_t smem;
};
constexpr size_t DENSE_SMEM = 208 * 1024; // the static arrays take up to 10 KB more

static int dense_stages(int k, size_t vb, int u)
{
    return (int)std::min<size_t>(DENSE_MAX_STAGES, (DENSE_SMEM - 2 * u * DW * DT * sizeof(double)) / ((size_t)k * DT * vb));
}

template <typename T>
static DenseForm dense_form(int k, int S)
{
    const int u = k <= 4 * DW ? 4 : (k <= 8 * DW && dense_stages(k, sizeof(T), 2) >= 6 ? 2 : 1);
    DenseForm f{};
    f.stages = dense_stages(k, sizeof(T), u);
    f.smem = (size_t)f.stages * k * DT * sizeof(T) + 2 * (size_t)u * DW * DT * sizeof(double);
    f.threads = dense_threads(u);
    dispatch_s(S, [&](auto SC) {
        if (k <= 4 * DW)
            f.kernel = (const void *)bb_dense_kernel<T, 4, SC.value, 4>;
        else if (k > 8 * DW)
            f.kernel = (const void *)bb_dense_kernel<T, 16, SC.value, 1>;
        else if (u == 2)
            f.kernel = (const void *)bb_dense_kernel<T, 8, SC.value, 2>;
        else
            f.kernel = (const void *)bb_dense_kernel<T, 8, SC.value, 1>;
    });
    return f;
}

// one block per SM, at most one per tile; 0: not for this shape
int dense_blocks(int k, int tiles, int S, int sms)
{
    if (k < 1 || k > DENSE_MAX_K || tiles < 1)
        return 0;
    for (const DenseForm &f : {dense_form<double>(k, S), dense_form<float>(k, S)}) {
        allow_shared(f.kernel, DENSE_SMEM);
        int per_sm = 0;
        CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f.kernel, f.threads, f.smem));
        if (per_sm < 1)
            return 0;
    }
    return std::min(sms, tiles);
}

void launch_bb_dense(int S, bool fp32, int blocks, const BBData &D, const BBParams &P, const DenseR &R,
                     const GridSlots &G, cudaStream_t s)
{
    DenseForm f = fp32 ? dense_form<float>(D.k, S) : dense_form<double>(D.k, S);
    void *args[] = {(void *)&D, (void *)&P, (void *)&R, (void *)&G, &f.stages};
    CK(cudaLaunchCooperativeKernel(f.kernel, blocks, f.threads, args, f.smem, s));
}

} // namespace pdhcg
