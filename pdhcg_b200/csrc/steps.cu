// steps.cu -- the step kernels (kernels.cuh) and their launchers.
#include "launch.cuh"

namespace pdhcg {

constexpr size_t PSD_STEP_SMEM = 200 * 1024;

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
// lane, the 3-slot blocks with one (mixed: both are done already); returns the
// number of launches.
template <typename T>
int launch_primal_cones(const StepData<T> &D, const StepParams &P, const ConeSplit &sp, int S, bool hasq, bool mixed,
                        cudaStream_t s)
{
    int launches = 0;
    if (sp.n_wide > 0 && !mixed) {
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
    if (sp.n_three > 0 && !mixed) {
        int grid = grid_for(sp.n_three, WARPS);
        if (hasq)
            primal_cone_kernel<1, T, true, CONES_THREE><<<grid, TPB, 0, s>>>(D, P, sp.three_d, sp.n_three);
        else
            primal_cone_kernel<1, T, false, CONES_THREE><<<grid, TPB, 0, s>>>(D, P, sp.three_d, sp.n_three);
        ++launches;
    }
    if (sp.n_psd > 0) { // LP path only: diagonal Q with PSD blocks takes the inner BB solve
        // a thread block per PSD block while the matrices fit in its shared
        // memory (order 112); a warp per block on global scratch beyond
        const size_t dyn = psd_work_doubles(D.psd_max) * sizeof(double);
        auto go = [&](auto kernel, int threads) {
            allow_shared(kernel, PSD_STEP_SMEM);
            kernel<<<grid_for(sp.n_psd, 1), threads, dyn, s>>>(D, P, sp.psd_d, sp.n_psd);
        };
        if (D.psd_max > 0 && dyn <= PSD_STEP_SMEM) {
            // 128 threads to order 20, 256 beyond: a round of order 20 is 255
            // updates and rotations for two barriers (us a step of 38 blocks, 128
            // and 256 threads: order 8 59 and 61, 16 130 and 131, 24 257 and 229,
            // 32 548 and 391)
            if (D.psd_max <= 20) {
                if (hasq)
                    go(psd_step_kernel<T, true, 128>, 128);
                else
                    go(psd_step_kernel<T, false, 128>, 128);
            } else {
                if (hasq)
                    go(psd_step_kernel<T, true, 256>, 256);
                else
                    go(psd_step_kernel<T, false, 256>, 256);
            }
        } else {
            dispatch_s(S, [&](auto SC) {
                int grid = grid_for(sp.n_psd, WARPS);
                if (hasq)
                    primal_cone_kernel<SC.value, T, true, CONES_PSD><<<grid, TPB, 0, s>>>(D, P, sp.psd_d, sp.n_psd);
                else
                    primal_cone_kernel<SC.value, T, false, CONES_PSD><<<grid, TPB, 0, s>>>(D, P, sp.psd_d, sp.n_psd);
            });
        }
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

// Free variables and cone blocks in one launch up to six thread blocks per SM,
// where the three launches would run one after the other for the length of
// their longest chains (us an iteration, one launch and three: 108 blocks 42
// and 59, 216 44 and 57, 324 45 and 61, 432 48 and 63, 863 56 and 68); beyond,
// where every kind fills the chip by itself, the kernels of one kind are
// leaner.  PSD and section blocks have launches of their own.  False: not for
// this problem, nothing launched.
template <typename T>
bool launch_primal_mixed(const StepData<T> &D, const StepParams &P, const ConeSplit &sp, int S, bool hasq,
                         cudaStream_t s)
{
    const int kinds = (D.n_free_tiles > 0) + (sp.n_wide > 0) + (sp.n_three > 0);
    if (kinds < 2 || !D.free_tiles && D.n_free > 0)
        return false;
    // (a warp per cone block, eight to a thread block, of either kind)
    const int fb = D.n_free > 0 ? grid_for(D.n_free_tiles, WARPS) : 0, wb = sp.n_wide > 0 ? grid_for(sp.n_wide, WARPS) : 0,
              tb = sp.n_three > 0 ? grid_for(sp.n_three, WARPS) : 0;
    if (fb + wb + tb > 6 * 148)
        return false;
    dispatch_s(sp.n_wide > 0 ? S : 1, [&](auto SC) {
        if (hasq)
            primal_mixed_kernel<SC.value, T, true><<<fb + wb + tb, TPB, 0, s>>>(D, P, fb, sp.wide_d, sp.n_wide, wb,
                                                                                 sp.three_d, sp.n_three);
        else
            primal_mixed_kernel<SC.value, T, false><<<fb + wb + tb, TPB, 0, s>>>(D, P, fb, sp.wide_d, sp.n_wide, wb,
                                                                                  sp.three_d, sp.n_three);
    });
    return true;
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
    template int launch_primal_cones<T>(const StepData<T> &, const StepParams &, const ConeSplit &, int, bool, bool,   \
                                        cudaStream_t);                                                                 \
    template bool launch_primal_mixed<T>(const StepData<T> &, const StepParams &, const ConeSplit &, int, bool,        \
                                         cudaStream_t);                                                                \
    template void launch_dual_cones<T>(const StepData<T> &, const StepParams &, int, cudaStream_t);                    \
    template void launch_dual_rows<T>(const StepData<T> &, const StepParams &, bool, bool, int, cudaStream_t);
PDHCG_STEP(double)
PDHCG_STEP(float)

} // namespace pdhcg
