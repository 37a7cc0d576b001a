// inner_impl.cuh -- launchers of the inner BB solve and the Q apply for one
// number G of lanes per row of Q (inner_g1.cu, inner_g4.cu, inner_g32.cu).
#pragma once

#include "launch.cuh"

namespace pdhcg {

// problems with fixed cone slots take the widest slot class (one
// instantiation per row group serves every block length)
template <int G>
const void *bb_kernel_of(int S, bool fixed, bool one_per_sm)
{
    const void *k = nullptr;
    if (fixed)
        k = (const void *)bb_kernel<G, 8, true, 1>;
    else
        dispatch_s(S, [&](auto SC) {
            k = one_per_sm ? (const void *)bb_kernel<G, SC.value, false, 1>
                           : (const void *)bb_kernel<G, SC.value, false, 2>;
        });
    return k;
}

template <int G>
int bb_blocks_per_sm_g(int S, bool fixed, bool one_per_sm)
{
    int a = 0, b = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, bb_kernel_of<G>(S, fixed, one_per_sm), TPB, 0));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, (const void *)q_apply_kernel<G>, TPB, 0));
    return std::min(a, b);
}

template <int G>
void launch_bb_g(int S, bool fixed, bool one_per_sm, int grid, const BBData &D, const BBParams &P, cudaStream_t s)
{
    void *args[] = {(void *)&D, (void *)&P};
    CK(cudaLaunchCooperativeKernel(bb_kernel_of<G>(S, fixed, one_per_sm), grid, TPB, args, 0, s));
}

template <int G>
void launch_q_apply_g(int grid, const BBData &D, const double *v, double *qx, cudaStream_t s)
{
    void *args[] = {(void *)&D, (void *)&v, (void *)&qx};
    CK(cudaLaunchCooperativeKernel((const void *)q_apply_kernel<G>, grid, TPB, args, 0, s));
}

#define PDHCG_INNER(G)                                                                                              \
    template int bb_blocks_per_sm_g<G>(int, bool, bool);                                                                  \
    template void launch_bb_g<G>(int, bool, bool, int, const BBData &, const BBParams &, cudaStream_t);               \
    template void launch_q_apply_g<G>(int, const BBData &, const double *, double *, cudaStream_t);

} // namespace pdhcg
