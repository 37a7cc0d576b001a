// project.cuh -- cone projections of a vector: the starting point of a solve
// and the kernel-level entry points.
#pragma once

#include "kernels.cuh"

namespace pdhcg {

// warp-per-cone projection of a vector (unit metric, d = rescaling);
// fixed: slots fixed by set_cone_fixed (NULL: none), sect: whether this
// block holds any (then the section projector, with warm start warm)
template <int S>
__device__ __forceinline__ void project_cone_block(int st, int L, int tp, double alpha, double *x, const double *d,
                                                   const double *q, double tau, int lane, double *psd,
                                                   const unsigned char *fixed = nullptr, bool sect = false,
                                                   double *warm = nullptr)
{
    WarpSlots<S> sl;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        sl.x[s] = i < L ? x[st + i] : 0.0;
        sl.d[s] = i < L ? d[st + i] : 1.0;
        sl.w[s] = (i < L && q) ? 1.0 + tau * q[st + i] : 1.0;
    }
    if (sect) {
        warp_section_project<S>(tp, sl, L, lane, section_bits<S>(fixed, st, L, lane), warm, alpha);
    } else {
        bool uni = warp_uniform_unit<S>(sl, L, lane);
        warp_project<S>(tp, sl, L, lane, uni, nullptr, alpha, psd);
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int i = lane + 32 * s;
        if (i < L)
            x[st + i] = sl.x[s];
    }
}

// psd_work / psd_off: PSD blocks' scratch and each block's offset in it
// (NULL: no PSD blocks)
template <int S>
__global__ void __launch_bounds__(TPB) project_cones_kernel(int ncones, const int *start, const int *len,
                                                            const int *type, const double *alpha, double *x,
                                                            const double *d, const double *q, double tau,
                                                            double *psd_work, const long long *psd_off,
                                                            const unsigned char *fixed = nullptr,
                                                            const unsigned char *cone_fixed = nullptr,
                                                            double *warm = nullptr)
{
    const int lane = threadIdx.x & 31;
    for (int cb = blockIdx.x * WARPS + (threadIdx.x >> 5); cb < ncones; cb += gridDim.x * WARPS) {
        const int st = start[cb], L = len[cb], tp = type[cb];
        const double a = alpha ? alpha[cb] : 0.0;
        double *psd = psd_work ? psd_work + psd_off[cb] : nullptr;
        const bool sect = cone_fixed && cone_fixed[cb];
        double *wb = warm ? warm + cb : nullptr;
        if (S > 1 && (tp == 2 || tp == 3)) // 3-slot blocks: the one-slot instantiation
            project_cone_block<1>(st, L, tp, a, x, d, q, tau, lane, psd, fixed, sect, wb);
        else if (tp == 4 && L > 32 * S) { // a long PSD block: in place, in memory (no metric)
            if (psd)
                warp_project_psd_mem(x + st, x + st, L, lane, psd);
        } else
            project_cone_block<S>(st, L, tp, a, x, d, q, tau, lane, psd, fixed, sect, wb);
    }
}

// every block a section block (pdhcg_b200_project_cone_sections)
template <int S>
__global__ void __launch_bounds__(TPB) project_sections_kernel(int ncones, const int *start, const int *len,
                                                               const int *type, const double *alpha, double *x,
                                                               const double *d, const double *q, double tau,
                                                               const unsigned char *fixed, double *warm)
{
    const int lane = threadIdx.x & 31;
    for (int cb = blockIdx.x * WARPS + (threadIdx.x >> 5); cb < ncones; cb += gridDim.x * WARPS) {
        const int st = start[cb], L = len[cb], tp = type[cb];
        const double a = alpha ? alpha[cb] : 0.0;
        double *wb = warm ? warm + cb : nullptr;
        if (S > 1 && (tp == 2 || tp == 3))
            project_cone_block<1>(st, L, tp, a, x, d, q, tau, lane, nullptr, fixed, true, wb);
        else
            project_cone_block<S>(st, L, tp, a, x, d, q, tau, lane, nullptr, fixed, true, wb);
    }
}

} // namespace pdhcg
