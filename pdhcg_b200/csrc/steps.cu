// steps.cu -- the step kernels (kernels.cuh) and their launchers.
#include "launch.cuh"

namespace pdhcg {

template <typename T>
void launch_primal_free(const StepData<T> &D, const StepParams &P, bool hasq, bool box_free, int grid, cudaStream_t s)
{
    if (hasq) {
        if (box_free)
            primal_free_kernel<T, true, false><<<grid, TPB, 0, s>>>(D, P);
        else
            primal_free_kernel<T, true, true><<<grid, TPB, 0, s>>>(D, P);
    } else {
        if (box_free)
            primal_free_kernel<T, false, false><<<grid, TPB, 0, s>>>(D, P);
        else
            primal_free_kernel<T, false, true><<<grid, TPB, 0, s>>>(D, P);
    }
}

// Primal step over the cone blocks: the SOC / RSOC blocks with S slots per
// lane, the 3-slot blocks with one; returns the number of launches.
template <typename T>
int launch_primal_cones(const StepData<T> &D, const StepParams &P, const ConeSplit &sp, int S, bool hasq,
                        cudaStream_t s)
{
    int launches = 0;
    if (sp.n_wide > 0) {
        // no more blocks than are resident at once: each warp then walks
        // several cone blocks and the warps drift apart, so one warp's
        // projection arithmetic overlaps other warps' loads (a full grid
        // starts every resident warp on its loads together); ~4 % of the
        // step on 20000 SOC blocks of 50
        dispatch_s(S, [&](auto SC) {
            if (hasq) {
                auto k = primal_cone_kernel<SC.value, T, true, CONES_WIDE>;
                int grid = std::min(grid_for(sp.n_wide, WARPS), resident_blocks((const void *)k));
                k<<<grid, TPB, 0, s>>>(D, P, sp.wide_d, sp.n_wide);
            } else {
                auto k = primal_cone_kernel<SC.value, T, false, CONES_WIDE>;
                int grid = std::min(grid_for(sp.n_wide, WARPS), resident_blocks((const void *)k));
                k<<<grid, TPB, 0, s>>>(D, P, sp.wide_d, sp.n_wide);
            }
        });
        ++launches;
    }
    if (sp.n_three > 0) {
        int grid = grid_for(sp.n_three, WARPS);
        if (hasq)
            primal_cone_kernel<1, T, true, CONES_THREE><<<grid, TPB, 0, s>>>(D, P, sp.three_d, sp.n_three);
        else
            primal_cone_kernel<1, T, false, CONES_THREE><<<grid, TPB, 0, s>>>(D, P, sp.three_d, sp.n_three);
        ++launches;
    }
    if (sp.n_psd > 0) { // LP path only: diagonal Q with PSD blocks takes the inner BB solve
        dispatch_s(S, [&](auto SC) {
            int grid = grid_for(sp.n_psd, WARPS);
            if (hasq)
                primal_cone_kernel<SC.value, T, true, CONES_PSD><<<grid, TPB, 0, s>>>(D, P, sp.psd_d, sp.n_psd);
            else
                primal_cone_kernel<SC.value, T, false, CONES_PSD><<<grid, TPB, 0, s>>>(D, P, sp.psd_d, sp.n_psd);
        });
        ++launches;
    }
    if (sp.n_sect > 0) { // blocks with fixed slots: section projectors, one slot class (any block length)
        int grid = grid_for(sp.n_sect, WARPS);
        if (hasq)
            primal_cone_kernel<8, T, true, CONES_SECTION><<<grid, TPB, 0, s>>>(D, P, sp.sect_d, sp.n_sect);
        else
            primal_cone_kernel<8, T, false, CONES_SECTION><<<grid, TPB, 0, s>>>(D, P, sp.sect_d, sp.n_sect);
        ++launches;
    }
    return launches;
}

template <typename T>
void launch_dual_cones(const StepData<T> &D, const StepParams &P, int S, cudaStream_t s)
{
    dispatch_s(S, [&](auto SC) {
        dual_cone_kernel<SC.value, T><<<grid_for(D.n_aff, WARPS), TPB, 0, s>>>(D, P);
    });
}

template <typename T>
void launch_dual_rows(const StepData<T> &D, const StepParams &P, bool eq_rows, bool has_g, int grid, cudaStream_t s)
{
    if (eq_rows) {
        if (has_g)
            dual_kernel<T, true, true><<<grid, TPB, 0, s>>>(D, P);
        else
            dual_kernel<T, true, false><<<grid, TPB, 0, s>>>(D, P);
    } else {
        if (has_g)
            dual_kernel<T, false, true><<<grid, TPB, 0, s>>>(D, P);
        else
            dual_kernel<T, false, false><<<grid, TPB, 0, s>>>(D, P);
    }
}

#define PDHCG_STEP(T)                                                                                                  \
    template void launch_primal_free<T>(const StepData<T> &, const StepParams &, bool, bool, int, cudaStream_t);       \
    template int launch_primal_cones<T>(const StepData<T> &, const StepParams &, const ConeSplit &, int, bool,         \
                                        cudaStream_t);                                                                 \
    template void launch_dual_cones<T>(const StepData<T> &, const StepParams &, int, cudaStream_t);                    \
    template void launch_dual_rows<T>(const StepData<T> &, const StepParams &, bool, bool, int, cudaStream_t);
PDHCG_STEP(double)
PDHCG_STEP(float)

} // namespace pdhcg
