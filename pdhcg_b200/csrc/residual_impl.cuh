// residual_impl.cuh -- launchers of the residual kernels (residual.cuh) for one
// storage type of the iterates (residual.cu, residual_f32.cu).
#pragma once

#include "launch.cuh"

namespace pdhcg {

// most dynamic shared memory of the two kernels: the scratch of the largest
// block held in registers for every warp; a thread block's for one PSD block
constexpr size_t RESIDUAL_SMEM = WARPS * psd_work_doubles(PSD_MAX_ORDER) * sizeof(double);
constexpr size_t RESIDUAL_PSD_SMEM = 190 * 1024;

template <typename VT>
void launch_residual(const ResidualData<VT> &D, const ResidualParams &P, int S, bool fixed, int blocks, cudaStream_t s)
{
    const size_t dyn = (size_t)D.psd_shared * WARPS * sizeof(double);
    auto go = [&](auto kernel) {
        if (dyn > 0)
            allow_shared(kernel, RESIDUAL_SMEM);
        kernel<<<blocks, TPB, dyn, s>>>(D, P);
    };
    if (fixed) // one slot class for problems with fixed cone slots
        go(residual_kernel<8, VT, true>);
    else
        dispatch_s(S, [&](auto SC) { go(residual_kernel<SC.value, VT, false>); });
}

inline size_t residual_psd_smem(int order)
{
    return (psd_work_doubles(order) + 3 * ((size_t)order * (order + 1) / 2)) * sizeof(double);
}

template <typename VT>
void launch_residual_psd(const ResidualData<VT> &D, const ResidualParams &P, const int *ids, int nids, int max_order,
                         int first, int blocks, cudaStream_t s)
{
    const size_t dyn = residual_psd_smem(max_order);
    allow_shared(residual_psd_kernel<VT>, RESIDUAL_PSD_SMEM);
    residual_psd_kernel<VT><<<blocks, TPB, dyn, s>>>(D, P, ids, nids, first);
}

} // namespace pdhcg
