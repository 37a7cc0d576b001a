// device.cuh -- device building blocks of the PDHCG-B200 kernels:
// warp/block reductions, CSR row products (stream mode for the hot kernels,
// row groups for set-up), and warp-cooperative weighted cone projections.
#pragma once

#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cuda_runtime.h>

namespace pdhcg {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o);
    return v; // identical in every lane: each butterfly step adds the same two operands
}

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmax(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

// |v| for an infinity-norm reduction: a non-finite entry makes the norm +inf
// (reference get_vector_inf_norm, src/utils.cu:548-567).
__device__ __forceinline__ double abs_or_inf(double v) { return isfinite(v) ? fabs(v) : INFINITY; }

// Sum of G consecutive lanes (G a power of two dividing 32).
template <int G>
__device__ __forceinline__ double group_sum(double v)
{
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
        v += __shfl_xor_sync(FULL, v, o, G);
    return v;
}

// sum_k val[k] * x[col[k]] over row r, G lanes cooperating (lane = lane in
// group); every lane of the warp must call it, ok == false gives 0 without
// reading the row.
template <int G, typename V>
__device__ __forceinline__ double row_dot(const int *__restrict__ rp, const int *__restrict__ ci,
                                          const V *__restrict__ val, const double *__restrict__ x, int r, int lane,
                                          bool ok = true)
{
    int b = ok ? __ldg(rp + r) : 0, e = ok ? __ldg(rp + r + 1) : 0;
    double s = 0.0;
    for (int k = b + lane; k < e; k += G)
        s += (double)__ldg(val + k) * __ldg(x + __ldg(ci + k));
    return group_sum<G>(s);
}

// Same with the vector held in FP32.
template <int G, typename V>
__device__ __forceinline__ double row_dot(const int *__restrict__ rp, const int *__restrict__ ci,
                                          const V *__restrict__ val, const float *__restrict__ x, int r, int lane,
                                          bool ok = true)
{
    int b = ok ? __ldg(rp + r) : 0, e = ok ? __ldg(rp + r + 1) : 0;
    double s = 0.0;
    for (int k = b + lane; k < e; k += G)
        s += (double)__ldg(val + k) * (double)__ldg(x + __ldg(ci + k));
    return group_sum<G>(s);
}

// ---------------------------------------------------------------------------
// Stream-mode CSR products for the hot step kernels.
//
// A warp owns up to 32 * S consecutive rows [r0, r0 + nr); lane l owns rows
// r0 + l + 32 s.  Their entries are one contiguous range [rp[r0], rp[r0+nr])
// of the CSR arrays, so the warp streams that range in chunks of
// STREAM_CHUNK entries: every lane issues STREAM_U independent coalesced
// loads of (col, val), then STREAM_U gathers of x, and stores the products in
// a per-warp shared buffer; each lane then adds the products of its own rows
// in entry order (the same order as a sequential row loop).
//
// A row longer than STREAM_ROW_MAX would leave one lane adding alone while
// the warp waits, so a warp whose rows include such a row reduces its rows
// one at a time across all 32 lanes instead (warp_sum; a different but
// fixed summation order).
// ---------------------------------------------------------------------------
#ifndef PDHCG_STREAM_U
#define PDHCG_STREAM_U 8
#endif
constexpr int STREAM_U = PDHCG_STREAM_U;
constexpr int STREAM_CHUNK = 32 * STREAM_U;
constexpr int STREAM_ROW_MAX = 64;

__device__ __forceinline__ int warp_max_int(int v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = max(v, __shfl_xor_sync(FULL, v, o));
    return v;
}

// ---------------------------------------------------------------------------
// Long rows.  A row of more than LONG_ROW entries (a dense constraint row, a
// variable in many rows) is too long for the stream mode below, and one warp
// per row would leave the product to the few warps whose tiles hold such
// rows.  So these rows are cut into segments of at most LONG_SEG entries:
// long_partials_kernel writes one partial product per segment (one warp
// each, fixed order), and the product that reads the row adds its
// segments' partials in segment order, each lane for its own row.  The
// partials belong to the last vector passed to that kernel: every product
// of a matrix with long rows is preceded by its pass.
//
// A segment whose columns are consecutive (a dense row, or a long dense part
// of one: budget and factor-exposure rows) is read without its column
// indices: seg_col holds its first column, -1 elsewhere.  That is 8 instead
// of 12 bytes per entry of a pass that HBM bounds, and the vector is read
// coalesced instead of gathered.
// ---------------------------------------------------------------------------
constexpr int LONG_ROW = STREAM_ROW_MAX; // every row beyond stream mode
constexpr int LONG_SEG = 4096;

struct LongRows {
    const int *rows;      // [n] long row ids, ascending
    const int *index;     // [rows of the matrix] a long row's index in rows, -1 for the others
    const int *seg_first; // [n + 1] first segment of each long row
    const int2 *seg;      // [nseg] entry range {begin, end} of each segment
    const int *seg_col;   // [nseg] first column of a segment of consecutive columns, else -1
    double *part;         // [nseg] partial products of the last pass
    int n, nseg;
};

// the same sum computed by the whole warp for one row (every lane calls it)
__device__ __forceinline__ double long_row_sum_warp(const LongRows &L, int row, int lane)
{
    const int i = __ldg(L.index + row);
    const int f = __ldg(L.seg_first + i), e = __ldg(L.seg_first + i + 1);
    double a = 0.0;
    for (int k = f + lane; k < e; k += 32)
        a += L.part[k];
    return warp_sum(a);
}

// sum of long row i's segment partials, in segment order (one lane)
__device__ __forceinline__ double long_row_fold(const LongRows &L, int i)
{
    const int f = __ldg(L.seg_first + i), e = __ldg(L.seg_first + i + 1);
    double a = 0.0;
    // eight partials' loads in flight, added in segment order
    int k = f;
    for (; k + 8 <= e; k += 8) {
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = L.part[k + u];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            a += v[u];
    }
    for (; k < e; ++k)
        a += L.part[k];
    return a;
}

// An entry of the vector of a product.  CG: the vector is written by other
// blocks of the same launch (persistent kernels), so the load goes to L2
// instead of the read-only path, which is not coherent within a launch.
template <bool CG, typename X>
__device__ __forceinline__ X load_x(const X *x)
{
    if constexpr (CG)
        return __ldcg(x);
    else
        return __ldg(x);
}

// one warp's dot product over entries [b, e), lane-strided, 4 partial sums
template <bool CG = false, typename V, typename X>
__device__ __forceinline__ double warp_range_dot(const int *__restrict__ ci, const V *__restrict__ val,
                                                 const X *__restrict__ x, int b, int e, int lane)
{
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    int k = b + lane;
    // two strides of 128 at a time: the eight index and value loads, then the
    // eight gathers, are in flight together; each partial sum still adds its
    // entries in stride order
    for (; k + 224 < e; k += 256) {
        int c[8];
        double v[8], w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            c[u] = __ldg(ci + k + 32 * u);
            v[u] = (double)__ldg(val + k + 32 * u);
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            w[u] = (double)load_x<CG>(x + c[u]);
        a0 += v[0] * w[0];
        a1 += v[1] * w[1];
        a2 += v[2] * w[2];
        a3 += v[3] * w[3];
        a0 += v[4] * w[4];
        a1 += v[5] * w[5];
        a2 += v[6] * w[6];
        a3 += v[7] * w[7];
    }
    for (; k + 96 < e; k += 128) {
        a0 += (double)__ldg(val + k) * (double)load_x<CG>(x + __ldg(ci + k));
        a1 += (double)__ldg(val + k + 32) * (double)load_x<CG>(x + __ldg(ci + k + 32));
        a2 += (double)__ldg(val + k + 64) * (double)load_x<CG>(x + __ldg(ci + k + 64));
        a3 += (double)__ldg(val + k + 96) * (double)load_x<CG>(x + __ldg(ci + k + 96));
    }
    // at most three strides remain (k + 96 >= e): their loads are issued
    // together, then added to a0 in stride order
    const bool p0 = k < e, p1 = k + 32 < e, p2 = k + 64 < e;
    const int c0 = p0 ? __ldg(ci + k) : 0, c1 = p1 ? __ldg(ci + k + 32) : 0, c2 = p2 ? __ldg(ci + k + 64) : 0;
    const double v0 = p0 ? (double)__ldg(val + k) : 0.0, v1 = p1 ? (double)__ldg(val + k + 32) : 0.0,
                 v2 = p2 ? (double)__ldg(val + k + 64) : 0.0;
    const double x0 = p0 ? (double)load_x<CG>(x + c0) : 0.0, x1 = p1 ? (double)load_x<CG>(x + c1) : 0.0,
                 x2 = p2 ? (double)load_x<CG>(x + c2) : 0.0;
    if (p0)
        a0 += v0 * x0;
    if (p1)
        a0 += v1 * x1;
    if (p2)
        a0 += v2 * x2;
    return warp_sum((a0 + a1) + (a2 + a3));
}

// the same over entries [b, e) whose columns are the consecutive ones from
// x's start on (x points at the first): no indices, two times eight loads in
// flight; the partial sums and their order are those of warp_range_dot
template <bool CG = false, typename V, typename X>
__device__ __forceinline__ double warp_range_dot_run(const V *__restrict__ val, const X *__restrict__ x, int len,
                                                     int lane)
{
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    int k = lane;
    for (; k + 480 < len; k += 512) {
        V v[16];
        X w[16];
#pragma unroll
        for (int u = 0; u < 16; ++u)
            v[u] = __ldg(val + k + 32 * u);
#pragma unroll
        for (int u = 0; u < 16; ++u)
            w[u] = load_x<CG>(x + k + 32 * u);
#pragma unroll
        for (int u = 0; u < 16; ++u)
            a[u & 3] += (double)v[u] * (double)w[u];
    }
    for (; k + 96 < len; k += 128)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            a[u] += (double)__ldg(val + k + 32 * u) * (double)load_x<CG>(x + k + 32 * u);
    for (; k < len; k += 32) // at most three strides
        a[0] += (double)__ldg(val + k) * (double)load_x<CG>(x + k);
    return warp_sum((a[0] + a[1]) + (a[2] + a[3]));
}

// the segment pass over warps gw, gw + nw, ... (a kernel body, or a phase
// of a cooperative kernel followed by a grid barrier)
template <bool CG = false, typename V, typename X>
__device__ __forceinline__ void long_partials(const LongRows &L, const int *__restrict__ ci,
                                              const V *__restrict__ val, const X *__restrict__ x, int gw, int nw,
                                              int lane)
{
    // the next segment's bounds are loaded before this segment's sum, so a
    // warp that walks many short segments does not wait for them each time
    int2 r = gw < L.nseg ? L.seg[gw] : make_int2(0, 0);
    int c = gw < L.nseg ? L.seg_col[gw] : -1;
    for (int sg = gw; sg < L.nseg; sg += nw) {
        const int2 rn = sg + nw < L.nseg ? L.seg[sg + nw] : make_int2(0, 0);
        const int cn = sg + nw < L.nseg ? L.seg_col[sg + nw] : -1;
        const double a = c >= 0 ? warp_range_dot_run<CG>(val + r.x, x + c, r.y - r.x, lane)
                                : warp_range_dot<CG>(ci, val, x, r.x, r.y, lane);
        if (lane == 0)
            L.part[sg] = a;
        r = rn;
        c = cn;
    }
}

template <typename V, typename X>
__global__ void __launch_bounds__(256) long_partials_kernel(LongRows L, const int *ci, const V *val, const X *x)
{
    long_partials(L, ci, val, x, (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5),
                  (int)((gridDim.x * blockDim.x) >> 5), (int)(threadIdx.x & 31));
}

// first column of every segment whose columns are consecutive, else -1; a
// warp per segment.  Short segments keep their indices (a run of them gains
// nothing over the gather).
constexpr int LONG_RUN_MIN = 256;

static __global__ void long_seg_col_kernel(LongRows L, const int *ci, int *seg_col)
{
    const int lane = threadIdx.x & 31;
    for (int sg = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); sg < L.nseg;
         sg += (int)((gridDim.x * blockDim.x) >> 5)) {
        const int2 r = L.seg[sg];
        const int c0 = ci[r.x];
        bool run = r.y - r.x >= LONG_RUN_MIN;
        if (run)
            for (int k = r.x + lane; k < r.y; k += 32)
                run = run && ci[k] == c0 + (k - r.x);
        run = __all_sync(FULL, run);
        if (lane == 0)
            seg_col[sg] = run ? c0 : -1;
    }
}

// number of rows longer than LONG_ROW entries
static __global__ void long_count_kernel(int rows, const int *rp, int *count)
{
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x)
        if (rp[r + 1] - rp[r] > LONG_ROW)
            atomicAdd(count, 1);
}

// out[s] = sum_k val[k] * x[ci[k]] over row r0 + lane + 32 s (0 when that
// row is past nr).  Every lane of the warp must call it with the same r0,
// nr (1 <= nr <= 32 S) and stage (STREAM_CHUNK doubles of this warp's
// shared memory).  Rows longer than LONG_ROW entries take their value from
// the segment partials of lr, which must hold this product's pass.  A tile
// holding such a row is otherwise reduced one row at a time by the whole
// warp (no table, lr.n = 0; or S > 2, where the lane-wise form would cost
// the wide cone kernels their registers).
template <int S, bool CG = false, typename V, typename X>
__device__ __forceinline__ void warp_stream_rows(const int *__restrict__ rp, const int *__restrict__ ci,
                                                 const V *__restrict__ val, const X *__restrict__ x, int r0, int nr,
                                                 int lane, double *stage, double (&out)[S], const LongRows &lr)
{
    int rb[S], re[S];
    int longest = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        rb[s] = re[s] = 0;
        if (i < nr) {
            rb[s] = __ldg(rp + r0 + i);
            re[s] = __ldg(rp + r0 + i + 1);
        }
        longest = max(longest, re[s] - rb[s]);
        out[s] = 0.0;
    }
    longest = warp_max_int(longest);
    const int b = __shfl_sync(FULL, rb[0], 0);
    int e = 0;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (s == ((nr - 1) >> 5))
            e = re[s];
    e = __shfl_sync(FULL, e, (nr - 1) & 31);

    if (longest <= STREAM_ROW_MAX) {
        for (int cb = b; cb < e; cb += STREAM_CHUNK) {
            int col[STREAM_U];
            double v[STREAM_U];
#pragma unroll
            for (int u = 0; u < STREAM_U; ++u) {
                const int k = cb + 32 * u + lane;
                col[u] = k < e ? __ldg(ci + k) : -1;
                v[u] = k < e ? (double)__ldg(val + k) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < STREAM_U; ++u)
                stage[32 * u + lane] = col[u] >= 0 ? v[u] * (double)load_x<CG>(x + col[u]) : 0.0;
            __syncwarp();
            const int ce = min(e, cb + STREAM_CHUNK);
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const int lo = max(rb[s], cb), hi = min(re[s], ce);
                double a = out[s];
                for (int k = lo; k < hi; ++k)
                    a += stage[k - cb];
                out[s] = a;
            }
            __syncwarp();
        }
    } else if (S <= 2 && lr.n > 0) {
        // every row longer than LONG_ROW is in lr: each lane folds its own
        // long row's partials or adds its own short row in entry order
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const bool valid = lane + 32 * s < nr;
            const bool lg = valid && re[s] - rb[s] > LONG_ROW;
            if (lg) {
                out[s] = long_row_fold(lr, __ldg(lr.index + r0 + lane + 32 * s));
            } else if (valid) {
                double a = 0.0;
                for (int k = rb[s]; k < re[s]; ++k)
                    a += (double)__ldg(val + k) * (double)load_x<CG>(x + __ldg(ci + k));
                out[s] = a;
            }
        }
    } else {
        for (int i = 0; i < nr; ++i) {
            int bi = 0, ei = 0;
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (s == (i >> 5)) {
                    bi = rb[s];
                    ei = re[s];
                }
            bi = __shfl_sync(FULL, bi, i & 31);
            ei = __shfl_sync(FULL, ei, i & 31);
            // (wide tiles with a long-row table: the warp folds each long row)
            const double a = (lr.n > 0 && ei - bi > LONG_ROW) ? long_row_sum_warp(lr, r0 + i, lane)
                                                                : warp_range_dot<CG>(ci, val, x, bi, ei, lane);
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (s == (i >> 5) && lane == (i & 31))
                    out[s] = a;
        }
    }
}

__device__ __forceinline__ double clampd(double lo, double x, double hi) { return fmax(lo, fmin(x, hi)); }

// ---------------------------------------------------------------------------
// Warp-cooperative cone projections.
//
// A warp owns one cone block of L slots; lane l holds slots l, l+32, ...
// in registers (S = slots per lane, compile time).  Inputs are the scaled
// candidate x (after the prox), the variable rescaling d and the metric
// weight w = 1 + tau q (w = 1 without a diagonal Q).  The cone is defined on
// u = x / d, so the projection minimises sum_i w_i d_i^2 (u_i - a_i)^2 with
// a_i = x_i / d_i (reference internal/cone_projection_utils.h:22-27).
// With d uniform and w == 1 the closed forms of the reference's thread
// kernels are used on x directly (src/kernels/pdhcg_soc_cone_kernels.cu:
// 296-324, src/kernels/pdhcg_rsoc_cone_kernels.cu:505-530); otherwise the
// multiplier of the KKT system is found by bracketed Newton, as in the
// reference's block kernels (pdhcg_soc_cone_kernels.cu:1725-2062,
// pdhcg_rsoc_cone_kernels.cu:2096-2631).  All lanes run the same scalar
// iteration on warp-reduced (bitwise identical) sums, so control flow is
// warp-uniform.
// ---------------------------------------------------------------------------

constexpr int ROOT_ITERS = 100;

template <int S>
struct WarpSlots {
    double x[S]; // in: candidate (scaled); out: projection (scaled)
    double d[S];
    double w[S];
};

// Standard SOC [v(k), w, z]: L = k + 2, apex slot index L-1.
// warm: this cone's multiplier from the previous call (NULL: none); on a
// root-finding exit the new multiplier is stored there (the reference keeps
// the same per-cone warm start, internal/internal_types.h:250).
template <int S>
__device__ void warp_project_soc(WarpSlots<S> &sl, int L, int lane, bool uniform_unit, double *warm)
{
    const int apex = L - 1;
    const int apex_lane = apex & 31, apex_s = apex >> 5;
    double xz = 0.0, dz = 1.0, wz = 1.0;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (s == apex_s) {
            xz = sl.x[s];
            dz = sl.d[s];
            wz = sl.w[s];
        }
    xz = __shfl_sync(FULL, xz, apex_lane);
    dz = __shfl_sync(FULL, dz, apex_lane);
    wz = __shfl_sync(FULL, wz, apex_lane);

    if (uniform_unit) {
        double ss = 0.0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            int i = lane + 32 * s;
            if (i < apex)
                ss += sl.x[s] * sl.x[s];
        }
        double r = sqrt(warp_sum(ss));
        if (r <= xz)
            return;
        if (r <= -xz) {
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < L)
                    sl.x[s] = 0.0;
            return;
        }
        double scale = (xz + r) / (2.0 * r);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            int i = lane + 32 * s;
            if (i < apex)
                sl.x[s] *= scale;
            else if (i == apex)
                sl.x[s] = scale * r;
        }
        return;
    }

    // u-space data: a = x / d, omega = w d^2; b = omega * a = w d x.  The
    // projection is u_i = b_i / (omega_i + lam), i.e. x_i = x_i omega_i / (omega_i + lam),
    // so the only per-slot reciprocals are 1/d (for the cone tests) and
    // 1/(omega_i + lam) (reused for the output).
    double b[S], om[S], inv[S];
    double n2 = 0.0, p2 = 0.0;
    // d uniform over the block (what cone-preserving scaling gives): one
    // reciprocal serves every slot (the same value each slot would compute)
    bool dsame = true;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < apex)
            dsame = dsame && sl.d[s] == dz;
    const double rdz = __all_sync(FULL, dsame) ? __drcp_rn(dz) : 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        b[s] = 0.0;
        om[s] = 1.0;
        inv[s] = 1.0;
        if (i < apex) {
            double rd = rdz != 0.0 ? rdz : __drcp_rn(sl.d[s]);
            double a = sl.x[s] * rd;
            om[s] = fmax(sl.w[s] * sl.d[s] * sl.d[s], DBL_MIN);
            b[s] = sl.w[s] * sl.d[s] * sl.x[s];
            n2 += a * a;
            p2 += b[s] * b[s];
        }
    }
    n2 = warp_sum(n2);
    p2 = warp_sum(p2);
    const double az = xz / dz;
    const double omz = fmax(wz * dz * dz, DBL_MIN);
    if (az >= 0.0 && n2 <= az * az)
        return; // inside
    if (-omz * az >= sqrt(p2)) { // -omega.a in the cone: apex
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < L)
                sl.x[s] = 0.0;
        return;
    }
    double lam, uz;
    if (az == 0.0) {
        lam = omz;
        double t2 = 0.0;
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < apex) {
                inv[s] = __drcp_rn(om[s] + lam);
                double t = b[s] * inv[s];
                t2 += t * t;
            }
        uz = sqrt(warp_sum(t2));
    } else {
        // f(lam) = |U|^2 - Z^2 with U_i = b_i/(om_i+lam), Z = omz az/(omz-lam);
        // root in (0, omz) when az > 0, in (omz, inf) when az < 0.
        const bool lower = az > 0.0;
        const double bz = omz * az;
        double lo = lower ? 0.0 : omz * (1.0 + 1e-14);
        double hi = lower ? omz * (1.0 - 1e-14) : INFINITY;
        double w0 = warm ? *warm : -1.0;
        lam = (w0 > lo && w0 < hi && isfinite(w0)) ? w0 : (lower ? 0.5 * (lo + hi) : 2.0 * omz);
        double izl = 0.0;
        bool done = false;
        for (int it = 0; it < ROOT_ITERS; ++it) {
            double t2 = 0.0;
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < apex) {
                    inv[s] = __drcp_rn(om[s] + lam);
                    double t = b[s] * inv[s];
                    t2 += t * t;
                }
            t2 = warp_sum(t2);
            izl = __drcp_rn(omz - lam);
            double z = bz * izl;
            double f = t2 - z * z;
            if ((lower && f > 0.0) || (!lower && f < 0.0))
                lo = lam;
            else
                hi = lam;
            if (fabs(f) <= 1e-13 * (1.0 + t2 + z * z) || (isfinite(hi) && hi - lo <= 1e-13 * (1.0 + hi + lo))) {
                done = true;
                break;
            }
            // f' only when a Newton step follows (a warm-started search
            // usually stops at its first evaluation)
            double dt2 = 0.0;
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < apex) {
                    double t = b[s] * inv[s];
                    dt2 += t * t * inv[s];
                }
            dt2 = warp_sum(dt2);
            double df = -2.0 * dt2 - 2.0 * z * z * izl;
            double nx = lam - f / df;
            // a Newton step below the resolution of lam cannot improve it:
            // stop there (without this, rounding that keeps |f| above its
            // tolerance sent the search into ~40 bisections of the bracket,
            // and the warp holding that block set the length of the launch)
            if (isfinite(nx) && fabs(nx - lam) <= 2.0 * DBL_EPSILON * fabs(lam)) {
                done = true;
                break;
            }
            if (!isfinite(nx) || !(nx > lo && nx < hi))
                nx = isfinite(hi) ? 0.5 * (lo + hi) : 2.0 * lam;
            lam = nx;
        }
        if (!done) { // iteration cap: inv and izl of the final lam
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < apex)
                    inv[s] = __drcp_rn(om[s] + lam);
            izl = __drcp_rn(omz - lam);
        }
        uz = bz * izl;
        if (warm && lane == 0)
            *warm = lam;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        if (i < apex)
            sl.x[s] = sl.x[s] * om[s] * inv[s];
        else if (i == apex)
            sl.x[s] = uz * dz;
    }
}

// Rotated SOC [v(k), s, t]: 2 s t >= |v|^2, s, t >= 0.  L = k + 2.
template <int S>
__device__ void warp_project_rsoc(WarpSlots<S> &sl, int L, int lane, bool uniform_unit, double *warm)
{
    const int is = L - 2, it_ = L - 1;
    double xs = 0.0, xt = 0.0, ds = 1.0, dt = 1.0, ws = 1.0, wt = 1.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        if (i == is) {
            xs = sl.x[s];
            ds = sl.d[s];
            ws = sl.w[s];
        }
        if (i == it_) {
            xt = sl.x[s];
            dt = sl.d[s];
            wt = sl.w[s];
        }
    }
    xs = __shfl_sync(FULL, xs, is & 31);
    ds = __shfl_sync(FULL, ds, is & 31);
    ws = __shfl_sync(FULL, ws, is & 31);
    xt = __shfl_sync(FULL, xt, it_ & 31);
    dt = __shfl_sync(FULL, dt, it_ & 31);
    wt = __shfl_sync(FULL, wt, it_ & 31);

    if (uniform_unit) {
        const double INV_SQRT2 = 0.7071067811865475;
        double wv = (xs - xt) * INV_SQRT2, zv = (xs + xt) * INV_SQRT2;
        double ss = 0.0;
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < is)
                ss += sl.x[s] * sl.x[s];
        double r = sqrt(wv * wv + warp_sum(ss));
        if (r <= zv)
            return;
        if (r <= -zv) {
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < L)
                    sl.x[s] = 0.0;
            return;
        }
        double scale = (zv + r) / (2.0 * r);
        double w_new = scale * wv, z_new = scale * r;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            int i = lane + 32 * s;
            if (i < is)
                sl.x[s] *= scale;
            else if (i == is)
                sl.x[s] = (z_new + w_new) * INV_SQRT2;
            else if (i == it_)
                sl.x[s] = (z_new - w_new) * INV_SQRT2;
        }
        return;
    }

    double a[S], om[S];
    double n2 = 0.0, p2 = 0.0, fobj = 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        a[s] = 0.0;
        om[s] = 1.0;
        if (i < is) {
            a[s] = sl.x[s] / sl.d[s];
            om[s] = fmax(sl.w[s] * sl.d[s] * sl.d[s], DBL_MIN);
            n2 += a[s] * a[s];
            p2 += (om[s] * a[s]) * (om[s] * a[s]);
            fobj += om[s] * a[s] * a[s];
        }
    }
    n2 = warp_sum(n2);
    p2 = warp_sum(p2);
    fobj = warp_sum(fobj);
    const double as = xs / ds, at = xt / dt;
    const double oms = fmax(ws * ds * ds, DBL_MIN), omt = fmax(wt * dt * dt, DBL_MIN);
    if (as >= 0.0 && at >= 0.0 && n2 <= 2.0 * as * at)
        return;
    const double bs = oms * as, bt = omt * at;
    if (bs <= 0.0 && bt <= 0.0 && p2 <= 2.0 * bs * bt) {
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < L)
                sl.x[s] = 0.0;
        return;
    }
    const double sqs = sqrt(oms), sqt = sqrt(omt), rm = sqs * sqt;
    const double balance = sqs * as + sqt * at;
    const double bscale = 1.0 + fabs(sqs * as) + fabs(sqt * at);
    double lam, ps, pt;
    if (fabs(balance) <= 64.0 * DBL_EPSILON * bscale) {
        lam = rm;
        double t2 = 0.0;
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < is) {
                double t = om[s] * a[s] / (om[s] + lam);
                t2 += t * t;
            }
        t2 = warp_sum(t2);
        double product = 0.5 * rm * t2, delta = sqs * as;
        double st = 0.5 * (-delta + sqrt(fmax(0.0, delta * delta + 4.0 * product)));
        ps = (st + delta) / sqs;
        pt = st / sqt;
    } else {
        // f(lam) = |U|^2 - 2 s t; root in (0, rm) when balance > 0, else (rm, inf)
        const bool lower = balance > 0.0;
        double lo = lower ? 0.0 : rm * (1.0 + 1e-14);
        double hi = lower ? rm * (1.0 - 1e-14) : INFINITY;
        double w0 = warm ? *warm : -1.0;
        lam = (w0 > lo && w0 < hi && isfinite(w0)) ? w0 : (lower ? 0.5 * (lo + hi) : 2.0 * rm);
        for (int itn = 0; itn < ROOT_ITERS; ++itn) {
            double t2 = 0.0, dt2 = 0.0;
#pragma unroll
            for (int s = 0; s < S; ++s)
                if (lane + 32 * s < is) {
                    double inv = 1.0 / (om[s] + lam);
                    double t = om[s] * a[s] * inv;
                    t2 += t * t;
                    dt2 += t * t * inv;
                }
            t2 = warp_sum(t2);
            dt2 = warp_sum(dt2);
            double idet = 1.0 / (oms * omt - lam * lam);
            double sv = omt * (oms * as + lam * at) * idet, tv = oms * (omt * at + lam * as) * idet;
            double f = INFINITY, df = -2.0 * dt2;
            if (sv >= 0.0 && tv >= 0.0) {
                f = t2 - 2.0 * sv * tv;
                double dsl = (omt * tv + lam * sv) * idet, dtl = (lam * tv + oms * sv) * idet;
                df -= 2.0 * (dsl * tv + sv * dtl);
            }
            if ((lower && f > 0.0) || (!lower && f < 0.0))
                lo = lam;
            else
                hi = lam;
            if (isfinite(f) && (fabs(f) <= 1e-13 * (1.0 + t2 + 2.0 * sv * tv) ||
                                (isfinite(hi) && hi - lo <= 1e-13 * (1.0 + hi + lo))))
                break;
            double nx = lam - f / df;
            if (isfinite(f) && isfinite(nx) && fabs(nx - lam) <= 2.0 * DBL_EPSILON * fabs(lam))
                break; // step below the resolution of lam (as for the SOC)
            if (!isfinite(nx) || !(nx > lo && nx < hi))
                nx = isfinite(hi) ? 0.5 * (lo + hi) : 2.0 * lam;
            lam = nx;
        }
        double det = oms * omt - lam * lam;
        ps = omt * (oms * as + lam * at) / det;
        pt = oms * (omt * at + lam * as) / det;
    }
    // axis candidates where the boundary is not smooth
    double sm = 0.0;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < is) {
            double v = om[s] * a[s] / (om[s] + lam);
            sm += om[s] * (v - a[s]) * (v - a[s]);
        }
    sm = warp_sum(sm) + oms * (ps - as) * (ps - as) + omt * (pt - at) * (pt - at);
    double s_axis = fmax(as, 0.0), t_axis = fmax(at, 0.0);
    double s_obj = fobj + oms * (s_axis - as) * (s_axis - as) + omt * at * at;
    double t_obj = fobj + oms * as * as + omt * (t_axis - at) * (t_axis - at);
    bool axis = false;
    if (s_obj < sm && s_obj <= t_obj) {
        axis = true;
        ps = s_axis;
        pt = 0.0;
    } else if (t_obj < sm) {
        axis = true;
        ps = 0.0;
        pt = t_axis;
    }
    if (warm && lane == 0 && !axis)
        *warm = lam;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        if (i < is)
            sl.x[s] = axis ? 0.0 : (om[s] * a[s] / (om[s] + lam)) * sl.d[s];
        else if (i == is)
            sl.x[s] = ps * ds;
        else if (i == it_)
            sl.x[s] = pt * dt;
    }
}

// ---------------------------------------------------------------------------
// Three-dimensional cones, projected by one thread.
//
// Exponential cone K = cl{(x, y, z) : y > 0, y exp(x / y) <= z}: the
// projection of r onto {v : v / d in K} in the unit metric of r's space,
// with the reference's sequence of tests and its Newton iteration on
// rho = x / y (src/kernels/pdhcg_exp_cone_kernels.cu:26-131): in-cone test,
// polar-cone test, the x <= 0, y <= 0 case, then at most 100 capped Newton
// steps with the same fallbacks.
// ---------------------------------------------------------------------------
__device__ inline void exp_cone_point(double r1, double r2, double r3, double d1, double d2, double d3, double &o1,
                                      double &o2, double &o3)
{
    const double a1 = r1 / d1, a2 = r2 / d2, a3 = r3 / d3;
    const bool inside = a2 > 0.0 ? (a1 / a2 < 700.0 && a2 * exp(a1 / a2) <= a3)
                                 : (a2 == 0.0 && a1 <= 0.0 && a3 >= 0.0);
    if (inside) {
        o1 = r1;
        o2 = r2;
        o3 = r3;
        return;
    }
    const bool polar = r1 > 0.0 ? ((d2 * r2) / (d1 * r1) < 700.0 &&
                                   d1 * r1 * exp((d2 * r2) / (d1 * r1)) + 2.718281828459045 * d3 * r3 <= 0.0)
                                : (r1 == 0.0 && r2 <= 0.0 && r3 <= 0.0);
    if (polar) {
        o1 = o2 = o3 = 0.0;
        return;
    }
    if (a1 <= 0.0 && a2 <= 0.0) {
        o1 = r1;
        o2 = 0.0;
        o3 = a3 < 0.0 ? 0.0 : r3;
        return;
    }
    const double al = (d3 / d1) * (d3 / d1), be = (d3 / d2) * (d3 / d2);
    double rho = 0.0;
    bool diverged = false;
    for (int it = 0; it < 100; ++it) {
        if (fabs(rho) >= 299.0) {
            diverged = true;
            break;
        }
        const double er = exp(rho), e2 = er * er, omr = 1.0 - rho;
        const double A = al - be * rho * omr, B = be * a1 * omr - al * a2;
        const double f = a1 - a2 * rho + a3 * er * A + e2 * B;
        const double df = -a2 + a3 * er * (A - be * (1.0 - 2.0 * rho)) + e2 * (2.0 * B - be * a1);
        if (fabs(df) < 1e-300)
            break;
        const double step = fmin(fmax(f / df, -10.0), 10.0);
        rho -= step;
        if (fabs(step) < 1e-13 * (1.0 + fabs(rho)))
            break;
    }
    const double er = exp(rho);
    const double u2 = (a1 + al * a3 * er) / (rho + al * er * er);
    if (diverged || !isfinite(u2) || u2 <= 0.0) {
        o1 = r1 < 0.0 ? r1 : 0.0;
        o2 = 0.0;
        o3 = r3 > 0.0 ? r3 : 0.0;
        return;
    }
    o1 = d1 * rho * u2;
    o2 = d2 * u2;
    o3 = d3 * u2 * er;
}

// Power cone K_a = {(x, y, z) : x, y >= 0, x^a y^(1-a) >= |z|}: weighted
// projection min sum w_i (v_i - r_i)^2 over K_a (reference
// src/kernels/pdhcg_power_cone_kernels.cu:25-133): in-cone and opposite-cone
// tests, then the root in log |v_z| with x, y the positive roots of the KKT
// quadratics, on the point scaled by its largest magnitude.
//
// The reference halves the bracket 80 times.  Each halving is a serial chain
// of an exp, square roots and two logs, and with one lane at work those 80
// chains set the length of the launch (76 us on 60 such blocks).  The warp
// instead tests 32 points of the bracket at once and keeps the interval
// between the last point below the root and the first above it, a factor of
// 33: four rounds narrow log DBL_MIN .. log |z| to 6e-4, from where Newton's
// method on the same function (kept inside the bracket) reaches the
// resolution of a double in about three steps.  If it has not after eight,
// further rounds narrow the bracket past it.
__device__ inline double pow_pos_root(double r, double q)
{
    if (!(q > 0.0))
        return fmax(r, 0.0);
    const double disc = sqrt(r * r + 4.0 * q); // |r| <= 1: the point is scaled
    return r >= 0.0 ? 0.5 * (r + disc) : (2.0 * q) / (disc - r);
}

// All lanes of the warp call it with the same block.
__device__ inline void pow_cone_point(double rx, double ry, double rz, double wx, double wy, double wz, double a,
                                      int lane, double &ox, double &oy, double &oz)
{
    double s = fmax(fabs(rx), fmax(fabs(ry), fabs(rz)));
    if (!(s > 0.0) || !isfinite(s))
        s = 1.0;
    rx /= s;
    ry /= s;
    rz /= s;
    const double az = fabs(rz), om = 1.0 - a;
    if (az == 0.0) {
        ox = fmax(rx, 0.0) * s;
        oy = fmax(ry, 0.0) * s;
        oz = 0.0;
        return;
    }
    if (rx > 0.0 && ry > 0.0 && a * log(rx) + om * log(ry) >= log(az)) {
        ox = rx * s;
        oy = ry * s;
        oz = rz * s;
        return;
    }
    if (rx <= 0.0 && ry <= 0.0) {
        const double u = rx < 0.0 ? (-wx * rx) / a : 0.0, v = ry < 0.0 ? (-wy * ry) / om : 0.0;
        if (u > 0.0 && v > 0.0 && a * log(u) + om * log(v) >= log(wz) + log(az)) {
            ox = oy = oz = 0.0;
            return;
        }
    }
    const double cx = 4.0 * a * (wz / wx), cy = 4.0 * om * (wz / wy);
    double lo = log(DBL_MIN), hi = log(az);
    if (!(hi > lo)) {
        ox = fmax(rx, 0.0) * s;
        oy = fmax(ry, 0.0) * s;
        oz = 0.0;
        return;
    }
    // one round: 32 points, the bracket a 33rd
    auto narrow = [&]() {
        const double w = (hi - lo) * (1.0 / 33.0);
        const double lr = lo + w * (lane + 1), rho = exp(lr);
        const double x = pow_pos_root(rx, 0.25 * cx * rho * (az - rho));
        const double y = pow_pos_root(ry, 0.25 * cy * rho * (az - rho));
        const bool below = x > 0.0 && y > 0.0 && a * log(x) + om * log(y) > lr;
        const unsigned above = ~__ballot_sync(FULL, below);
        const int c = above ? __ffs(above) - 1 : 32; // points below the root
        const double l2 = c > 0 ? lo + w * c : lo, h2 = c < 32 ? lo + w * (c + 1) : hi;
        const bool moved = h2 - l2 < hi - lo;
        lo = l2;
        hi = h2;
        return moved;
    };
    bool more = true;
    for (int it = 0; more && it < 4; ++it)
        more = narrow();
    // Newton on f(lr) = a log x + om log y - lr, every lane alike
    double lr = lo + 0.5 * (hi - lo);
    bool done = false;
    for (int it = 0; more && !done && it < 8; ++it) {
        const double rho = exp(lr), qs = 0.25 * rho * (az - rho), dq = 0.25 * rho * (az - 2.0 * rho);
        const double x = pow_pos_root(rx, cx * qs), y = pow_pos_root(ry, cy * qs);
        if (!(x > 0.0 && y > 0.0 && qs > 0.0))
            break;
        const double f = a * log(x) + om * log(y) - lr;
        if (f > 0.0)
            lo = lr;
        else
            hi = lr;
        // x' = cx dq / (2 x - rx): x^2 - rx x = cx qs
        const double df = a * cx * dq / ((2.0 * x - rx) * x) + om * cy * dq / ((2.0 * y - ry) * y) - 1.0;
        const double nx = lr - f / df;
        if (!(nx > lo && nx < hi)) {
            // outside the bracket: at the resolution of lr the bracket has closed on it
            done = fabs(f / df) <= 4.0 * DBL_EPSILON * (1.0 + fabs(lr));
            if (!done && !isfinite(nx))
                break;
            lr = done ? lr : lo + 0.5 * (hi - lo);
            continue;
        }
        done = fabs(nx - lr) <= 4.0 * DBL_EPSILON * (1.0 + fabs(lr));
        lr = nx;
    }
    if (!done) {
        for (int it = 0; more && it < 13; ++it)
            more = narrow();
        lr = lo + 0.5 * (hi - lo);
    }
    const double rho = exp(lr);
    const double x = pow_pos_root(rx, 0.25 * cx * rho * (az - rho));
    const double y = pow_pos_root(ry, 0.25 * cy * rho * (az - rho));
    ox = x * s;
    oy = y * s;
    oz = (rz >= 0.0 ? 1.0 : -1.0) * fmin(rho, exp(a * log(x) + om * log(y))) * s;
}

// A 3-slot block held in lanes 0..2 (S = 1 slot each), metric w, scaling d:
// an exponential block (type 2) is projected by lane 0, a power block (type
// 3) by the whole warp; the result goes back to the three lanes.  Only the
// one-slot (S = 1) instantiations of the cone-block bodies reach it, so its
// loops stay out of the wide SOC bodies' register allocation.
template <int S>
__device__ __forceinline__ void warp_project3(int type, WarpSlots<S> &sl, int lane, double alpha)
{
    double3 x, d, w;
    x.x = __shfl_sync(FULL, sl.x[0], 0);
    x.y = __shfl_sync(FULL, sl.x[0], 1);
    x.z = __shfl_sync(FULL, sl.x[0], 2);
    d.x = __shfl_sync(FULL, sl.d[0], 0);
    d.y = __shfl_sync(FULL, sl.d[0], 1);
    d.z = __shfl_sync(FULL, sl.d[0], 2);
    w.x = __shfl_sync(FULL, sl.w[0], 0);
    w.y = __shfl_sync(FULL, sl.w[0], 1);
    w.z = __shfl_sync(FULL, sl.w[0], 2);
    double3 o = make_double3(0.0, 0.0, 0.0);
    if (type == 2) {
        if (lane == 0) { // the sqrt(w) change of variables
            const double s0 = sqrt(w.x > 0.0 ? w.x : 1.0), s1 = sqrt(w.y > 0.0 ? w.y : 1.0),
                         s2 = sqrt(w.z > 0.0 ? w.z : 1.0);
            exp_cone_point(s0 * x.x, s1 * x.y, s2 * x.z, s0 * d.x, s1 * d.y, s2 * d.z, o.x, o.y, o.z);
            o.x /= s0;
            o.y /= s1;
            o.z /= s2;
        }
        o.x = __shfl_sync(FULL, o.x, 0);
        o.y = __shfl_sync(FULL, o.y, 0);
        o.z = __shfl_sync(FULL, o.z, 0);
    } else { // scaled space, weights w d^2
        pow_cone_point(x.x / d.x, x.y / d.y, x.z / d.z, w.x * d.x * d.x, w.y * d.y * d.y, w.z * d.z * d.z, alpha, lane,
                       o.x, o.y, o.z);
        o.x *= d.x;
        o.y *= d.y;
        o.z *= d.z;
    }
    if (lane < 3)
        sl.x[0] = lane == 0 ? o.x : (lane == 1 ? o.y : o.z);
}

// Cone kinds an instantiation carries: SOC / RSOC (any S), and the 3-slot
// exponential / power cones (S = 1 only; callers route those blocks there).
// ---------------------------------------------------------------------------
// PSD blocks.  The block's L = n (n + 1) / 2 slots hold svec(X): the lower
// triangle down the columns, off-diagonal entries scaled by sqrt 2 (the
// reference's packing, src/kernels/pdhcg_psd_cone_kernels.cu:65-91).  The
// projection is the Frobenius one in the scaled space, as the reference
// takes it (:415-475; no metric): the warp unpacks X into work[0, n^2)
// (this block's device scratch), diagonalises it by Jacobi rotations while
// accumulating the eigenvectors in work[n^2, 2 n^2), clips the negative
// eigenvalues and repacks.
//
// A sweep visits the pairs in round-robin order (the tournament ordering of
// Brent and Luk 1985): n - 1 rounds (n for odd n) of n / 2 disjoint pairs.  A
// round's rotations are independent, so lane i computes the angle of pair
// i, and the two-sided update splits into 2 x 2 blocks (pair i's rows,
// pair j's columns) that each read and write only themselves: one barrier
// between the angles and the update, one after it.  Visiting the pairs one
// at a time instead (n (n - 1) / 2 angle computations in series, each some
// 600 cycles of divisions and square roots, and four barriers) took 2 ms for
// a block of order 20.  The rotation is Rutishauser's; the search stops when
// the off-diagonal mass is below 1e-28 of the whole (at most 100 sweeps).
// Blocks of order up to PSD_MAX_ORDER (L <= 256 slots) are held in the warp's
// registers between the steps, longer ones in memory.
// ---------------------------------------------------------------------------
constexpr int PSD_MAX_ORDER = 22;
constexpr int PSD_MAX_SWEEPS = 100;
constexpr double PSD_OFF_REL = 1e-28;

// (row, col) of svec slot i of an order-n block: column c starts at slot
// c n - c (c - 1) / 2
__device__ __forceinline__ void psd_slot_rc(int i, int n, int &row, int &col)
{
    const float b = 2.0f * (float)n + 1.0f;
    int c = max(0, min(n - 1, (int)((b - sqrtf(fmaxf(b * b - 8.0f * (float)i, 0.0f))) * 0.5f)));
    while (c > 0 && i < c * n - c * (c - 1) / 2)
        --c;
    while (i >= (c + 1) * n - (c + 1) * c / 2)
        ++c;
    col = c;
    row = c + (i - (c * n - c * (c - 1) / 2));
}

// Scratch of one block in doubles: A, the eigenvectors (V^T, one per row),
// and the cosine and sine of each pair of a round.
__host__ __device__ constexpr long long psd_work_doubles(long long order)
{
    return 2 * order * order + 2 * ((order + 1) / 2);
}

// Rotation for a pair: the tangent of the smaller angle that annihilates a_pq
// is t = a2 / (h + sign(h) sqrt(h^2 + a2^2)), h = a_qq - a_pp, a2 = 2 a_pq.
// The rounds are chains of these angles, and FP64 square roots and divisions
// are a few hundred cycles each, so t starts from its FP32 value on the pair
// scaled by its larger magnitude (a power of two) and takes one Newton step in
// FP64 on t^2 a2 / 2 + t h - a2 / 2 (error 3e-7, then 1e-13; the slope at the root
// is that square root, and its reciprocal may be FP32, as it multiplies a
// correction of 3e-7), and the cosine,
// which makes (c, t c) a rotation to FP64 rounding, is 1 / sqrt(1 + t^2) by two
// Newton steps from its FP32 value (errors 1e-7, 1e-14, below rounding).  What
// the angle leaves of a_pq is kept, not set to zero.
__device__ __forceinline__ void jacobi_angle(double app, double aqq, double apq, double &c, double &sn)
{
    c = 1.0;
    sn = 0.0;
    const double h = aqq - app, a2 = 2.0 * apq, mag = fmax(fabs(h), fabs(a2));
    if (!(mag > 0.0) || !(mag < 8e307)) // nothing to rotate (or out of range)
        return;
    // 2^-e with e the exponent of mag (a subnormal pair is left as it is)
    const int e = (int)((__double_as_longlong(mag) >> 52) & 0x7ff);
    if (e < 2 || e > 2045)
        return;
    const double scale = __longlong_as_double((long long)(2046 - e) << 52);
    const double hs = h * scale, as = a2 * scale;
    const float hf = (float)hs, af = (float)as;
    const float q = hf * hf + af * af, rq = copysignf(rsqrtf(q), hf); // q in [1, 8)
    const double t0 = (double)__fdividef(af, hf + q * rq);
    const double t = fma(-(double)rq, fma(fma(0.5 * as, t0, hs), t0, -0.5 * as), t0);
    const double r = fma(t, t, 1.0);
    double y = (double)rsqrtf((float)r);
    y = y * fma(-0.5 * r * y, y, 1.5);
    y = y * fma(-0.5 * r * y, y, 1.5);
    c = y;
    sn = t * y;
}

// pair i of round r over m players: {m - 1, r}, then {r + i, r - i} modulo m - 1
__device__ __forceinline__ void jacobi_pair(int m, int r, int i, int &p, int &q)
{
    int a = m - 1, b = r;
    if (i > 0) {
        a = r + i;
        b = r - i;
        if (a >= m - 1)
            a -= m - 1;
        if (b < 0)
            b += m - 1;
    }
    p = min(a, b);
    q = max(a, b);
}

// (i, j), i <= j, of index t of the upper triangle, columns in order
__device__ __forceinline__ void jacobi_block(int t, int &i, int &j)
{
    j = (int)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while ((j + 1) * (j + 2) / 2 <= t)
        ++j;
    while (j * (j + 1) / 2 > t)
        --j;
    i = t - j * (j + 1) / 2;
}

// A <- J' A J on the rows of pair i and the columns of pair j (i <= j; an
// index n is the bye of an odd order) and on the mirror image
__device__ __forceinline__ void jacobi_update(double *A, int n, int m, int r, int i, int j, const double *cs)
{
    int pi, qi, pj, qj;
    jacobi_pair(m, r, i, pi, qi);
    jacobi_pair(m, r, j, pj, qj);
    const double ci = cs[2 * i], si = cs[2 * i + 1], cj = cs[2 * j], sj = cs[2 * j + 1];
    const bool fi = qi < n, fj = qj < n;
    const double app = A[(size_t)pi * n + pj], apq = fj ? A[(size_t)pi * n + qj] : 0.0;
    const double aqp = fi ? A[(size_t)qi * n + pj] : 0.0, aqq = fi && fj ? A[(size_t)qi * n + qj] : 0.0;
    // columns by pair j, then rows by pair i
    const double bpp = cj * app - sj * apq, bpq = sj * app + cj * apq;
    const double bqp = cj * aqp - sj * aqq, bqq = sj * aqp + cj * aqq;
    const double dpp = ci * bpp - si * bqp, dqp = si * bpp + ci * bqp;
    const double dpq = ci * bpq - si * bqq, dqq = si * bpq + ci * bqq;
    if (i == j) { // the rotated pair itself
        A[(size_t)pi * n + pi] = dpp;
        if (fi) {
            const double off = 0.5 * (dpq + dqp); // what the angle's rounding left
            A[(size_t)qi * n + qi] = dqq;
            A[(size_t)pi * n + qi] = off;
            A[(size_t)qi * n + pi] = off;
        }
        return;
    }
    A[(size_t)pi * n + pj] = dpp;
    A[(size_t)pj * n + pi] = dpp;
    if (fj) {
        A[(size_t)pi * n + qj] = dpq;
        A[(size_t)qj * n + pi] = dpq;
    }
    if (fi) {
        A[(size_t)qi * n + pj] = dqp;
        A[(size_t)pj * n + qi] = dqp;
    }
    if (fi && fj) {
        A[(size_t)qi * n + qj] = dqq;
        A[(size_t)qj * n + qi] = dqq;
    }
}

// Diagonalises the symmetric n x n matrix A (full, row-major) in place by
// round-robin Jacobi; row e of Vt receives the e-th eigenvector.  Every lane
// of the warp calls it; A is visible to all of them.
__device__ inline void warp_jacobi(double *A, double *Vt, double *cs, int n, int lane)
{
    for (int e = lane; e < n * n; e += 32)
        Vt[e] = (e / n == e % n) ? 1.0 : 0.0;
    __syncwarp();
    const int m = n + (n & 1), np = m / 2; // odd n: index n is a bye
    for (int sweep = 0; sweep < PSD_MAX_SWEEPS; ++sweep) {
        double off = 0.0, all = 0.0;
        for (int r = 0; r < n; ++r)
            for (int k = lane; k < n; k += 32) {
                const double a = A[(size_t)r * n + k], a2 = a * a;
                all += a2;
                if (k != r)
                    off += a2;
            }
        off = warp_sum(off);
        all = warp_sum(all);
        if (!(off > PSD_OFF_REL * all))
            break;
        for (int r = 0; r < m - 1; ++r) {
            for (int i = lane; i < np; i += 32) {
                int p, q;
                jacobi_pair(m, r, i, p, q);
                double c = 1.0, sn = 0.0;
                if (q < n)
                    jacobi_angle(A[(size_t)p * n + p], A[(size_t)q * n + q], A[(size_t)p * n + q], c, sn);
                cs[2 * i] = c;
                cs[2 * i + 1] = sn;
            }
            __syncwarp();
            for (int t = lane; t < np * (np + 1) / 2; t += 32) {
                int i, j;
                jacobi_block(t, i, j);
                jacobi_update(A, n, m, r, i, j, cs);
            }
            for (int j = 0; j < np; ++j) {
                int p, q;
                jacobi_pair(m, r, j, p, q);
                if (q >= n)
                    continue;
                const double c = cs[2 * j], sn = cs[2 * j + 1];
                for (int k = lane; k < n; k += 32) {
                    const double vp = Vt[(size_t)p * n + k], vq = Vt[(size_t)q * n + k];
                    Vt[(size_t)p * n + k] = c * vp - sn * vq;
                    Vt[(size_t)q * n + k] = sn * vp + c * vq;
                }
            }
            __syncwarp();
        }
    }
}

// The same by a block of NT threads, A, Vt and cs in its shared memory; red:
// 2 NT / 32 doubles.  A round's work is spread so thin over the warps (order
// 20: 10 angles, 55 blocks, 200 rotated eigenvector entries) that its length
// is one angle and one update's latency.
template <int NT>
__device__ inline void cta_jacobi(double *A, double *Vt, double *cs, double *red, int n)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int e = tid; e < n * n; e += NT)
        Vt[e] = (e / n == e % n) ? 1.0 : 0.0;
    const int m = n + (n & 1), np = m / 2, nblk = np * (np + 1) / 2, nv = np * n;
    int i0 = 0, j0 = 0; // this thread's first block and eigenvector entry
    if (tid < nblk)
        jacobi_block(tid, i0, j0);
    const int vj0 = tid / n, vk0 = tid - vj0 * n;
    __syncthreads();
    for (int sweep = 0; sweep < PSD_MAX_SWEEPS; ++sweep) {
        double off = 0.0, all = 0.0;
        for (int e = tid; e < n * n; e += NT) {
            const double a2 = A[e] * A[e];
            all += a2;
            if (e / n != e % n)
                off += a2;
        }
        off = warp_sum(off);
        all = warp_sum(all);
        if (lane == 0) {
            red[2 * warp] = off;
            red[2 * warp + 1] = all;
        }
        __syncthreads();
        off = all = 0.0;
        for (int w = 0; w < NT / 32; ++w) {
            off += red[2 * w];
            all += red[2 * w + 1];
        }
        if (!(off > PSD_OFF_REL * all))
            break;
        for (int r = 0; r < m - 1; ++r) {
            for (int i = tid; i < np; i += NT) {
                int p, q;
                jacobi_pair(m, r, i, p, q);
                double c = 1.0, sn = 0.0;
                if (q < n)
                    jacobi_angle(A[p * n + p], A[q * n + q], A[p * n + q], c, sn);
                cs[2 * i] = c;
                cs[2 * i + 1] = sn;
            }
            __syncthreads();
            for (int t = tid; t < nv; t += NT) {
                int j = vj0, k = vk0;
                if (t != tid) {
                    j = t / n;
                    k = t - j * n;
                }
                int p, q;
                jacobi_pair(m, r, j, p, q);
                if (q < n) {
                    const double c = cs[2 * j], sn = cs[2 * j + 1], vp = Vt[p * n + k], vq = Vt[q * n + k];
                    Vt[p * n + k] = c * vp - sn * vq;
                    Vt[q * n + k] = sn * vp + c * vq;
                }
            }
            for (int t = tid; t < nblk; t += NT) {
                int i = i0, j = j0;
                if (t != tid)
                    jacobi_block(t, i, j);
                jacobi_update(A, n, m, r, i, j, cs);
            }
            __syncthreads();
        }
    }
}

template <int S>
__device__ void warp_project_psd(WarpSlots<S> &sl, int L, int lane, double *work)
{
    int n = 0;
    while (n * (n + 1) / 2 < L)
        ++n;
    if (n == 1) {
        if (lane == 0)
            sl.x[0] = fmax(sl.x[0], 0.0);
        return;
    }
    bool finite = true;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < L)
            finite &= isfinite(sl.x[s]) != 0;
    if (!__all_sync(FULL, finite)) { // the reference's failed decomposition gives NaN
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (lane + 32 * s < L)
                sl.x[s] = __longlong_as_double(0x7ff8000000000000LL);
        return;
    }
    const double R2 = 1.41421356237309504880, IR2 = 0.70710678118654752440;
    double *A = work, *Vt = work + n * n;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        if (i < L) {
            int row, col;
            psd_slot_rc(i, n, row, col);
            const double v = row == col ? sl.x[s] : sl.x[s] * IR2;
            A[row * n + col] = v;
            A[col * n + row] = v;
        }
    }
    __syncwarp();
    warp_jacobi(A, Vt, work + 2 * n * n, n, lane);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const int i = lane + 32 * s;
        if (i < L) {
            int row, col;
            psd_slot_rc(i, n, row, col);
            double v = 0.0;
            for (int e = 0; e < n; ++e)
                v += fmax(A[e * n + e], 0.0) * Vt[e * n + row] * Vt[e * n + col];
            sl.x[s] = row == col ? v : v * R2;
        }
    }
    __syncwarp(); // the scratch may be reused by this warp's next projection
}

// PSD blocks of any order ("long" blocks: more slots than a warp's
// registers hold, L > 32 S).  The svec lies in memory (in, L doubles; out
// may alias it); the warp unpacks it into work[0, n^2), diagonalises it as
// above, clips and repacks into out.  Callers stage the block's candidate in
// its scratch (psd_stage, after the decomposition's doubles) and call this
// instead of the register form.
__device__ __forceinline__ int psd_order(int L)
{
    int n = (int)floor(sqrt(2.0 * L));
    while (n * (n + 1) / 2 < L)
        ++n;
    while (n > 1 && (n - 1) * n / 2 >= L)
        --n;
    return n;
}

__device__ __forceinline__ double *psd_stage(double *work, int n) { return work + psd_work_doubles(n); }

// a block's whole scratch: L doubles of candidate staging per long block,
// after the decomposition's (the residual stages three vectors, so 3 L are
// kept)
__host__ __device__ inline long long psd_scratch_doubles(int order, bool is_long)
{
    const long long L = (long long)order * (order + 1) / 2;
    return psd_work_doubles(order) + (is_long ? 3 * L : 0);
}

__device__ inline void warp_project_psd_mem(const double *in, double *out, int L, int lane, double *work)
{
    const int n = psd_order(L);
    if (n == 1) {
        if (lane == 0)
            out[0] = fmax(in[0], 0.0);
        __syncwarp();
        return;
    }
    bool finite = true;
    for (int i = lane; i < L; i += 32)
        finite &= isfinite(in[i]) != 0;
    if (!__all_sync(FULL, finite)) { // the reference's failed decomposition gives NaN
        for (int i = lane; i < L; i += 32)
            out[i] = __longlong_as_double(0x7ff8000000000000LL);
        __syncwarp();
        return;
    }
    const double R2 = 1.41421356237309504880, IR2 = 0.70710678118654752440;
    double *A = work, *Vt = work + (size_t)n * n;
    for (int col = 0, first = 0; col < n; first += n - col, ++col)
        for (int row = col + lane; row < n; row += 32) {
            const double x = in[first + row - col];
            const double v = row == col ? x : x * IR2;
            A[(size_t)row * n + col] = v;
            A[(size_t)col * n + row] = v;
        }
    __syncwarp();
    warp_jacobi(A, Vt, work + 2 * (size_t)n * n, n, lane);
    for (int col = 0, first = 0; col < n; first += n - col, ++col)
        for (int row = col + lane; row < n; row += 32) {
            double v = 0.0;
            for (int e = 0; e < n; ++e)
                v += fmax(A[(size_t)e * n + e], 0.0) * Vt[(size_t)e * n + row] * Vt[(size_t)e * n + col];
            out[first + row - col] = row == col ? v : v * R2;
        }
    __syncwarp(); // the scratch and out may be read by other lanes next
}

// Cone kinds an instantiation carries: SOC / RSOC (any S), the 3-slot
// exponential / power cones (S = 1 only; callers route those blocks there)
// and PSD blocks (psd: this block's scratch).  Blocks with
// fixed slots (any type but PSD) are a launch class of their own,
// CONES_SECTION, projected by section.cuh.
enum ConeKinds { CONES_WIDE = 1, CONES_THREE = 2, CONES_PSD = 4, CONES_ALL = 7, CONES_SECTION = 8 };

template <int S, int KINDS = CONES_ALL>
__device__ __forceinline__ void warp_project(int type, WarpSlots<S> &sl, int L, int lane, bool uniform_unit,
                                             double *warm, double alpha = 0.0, double *psd = nullptr)
{
    if ((KINDS & CONES_WIDE) && type == 1) // CONE_STANDARD_SOC
        warp_project_soc<S>(sl, L, lane, uniform_unit, warm);
    else if ((KINDS & CONES_WIDE) && type == 0) // CONE_ROTATED_SOC
        warp_project_rsoc<S>(sl, L, lane, uniform_unit, warm);
    else if ((KINDS & CONES_THREE) && S == 1 && (type == 2 || type == 3)) // CONE_EXPONENTIAL, CONE_POWER
        warp_project3<S>(type, sl, lane, alpha);
    else if ((KINDS & CONES_PSD) && type == 4 && psd != nullptr) // CONE_PSD
        warp_project_psd<S>(sl, L, lane, psd);
}

// Is d uniform over the block and w == 1 everywhere?  (warp vote)
template <int S>
__device__ __forceinline__ bool warp_uniform_unit(const WarpSlots<S> &sl, int L, int lane)
{
    double d0 = __shfl_sync(FULL, sl.d[0], 0);
    bool ok = true;
#pragma unroll
    for (int s = 0; s < S; ++s)
        if (lane + 32 * s < L)
            ok = ok && (sl.d[s] == d0) && (sl.w[s] == 1.0);
    return __all_sync(FULL, ok);
}

} // namespace pdhcg
