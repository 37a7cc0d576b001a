// inner.cu -- the inner BB solve and the Q apply by lanes per row of Q.
#include "launch.cuh"

namespace pdhcg {

template <int G>
int bb_blocks_per_sm_g(int S, bool fixed, bool one_per_sm);
template <int G>
void launch_bb_g(int S, bool fixed, bool one_per_sm, int grid, const BBData &D, const BBParams &P, cudaStream_t s);
template <int G>
void launch_q_apply_g(int grid, const BBData &D, const double *v, double *qx, cudaStream_t s);

int bb_blocks_per_sm(int G, int S, bool fixed, bool one_per_sm)
{
    int r = 0;
    dispatch_rg(G, [&](auto GC) { r = bb_blocks_per_sm_g<GC.value>(S, fixed, one_per_sm); });
    return r;
}

void launch_bb(int G, int S, bool fixed, bool one_per_sm, int grid, const BBData &D, const BBParams &P, cudaStream_t s)
{
    dispatch_rg(G, [&](auto GC) { launch_bb_g<GC.value>(S, fixed, one_per_sm, grid, D, P, s); });
}

void launch_q_apply(int G, int grid, const BBData &D, const double *v, double *qx, cudaStream_t s)
{
    dispatch_rg(G, [&](auto GC) { launch_q_apply_g<GC.value>(grid, D, v, qx, s); });
}

} // namespace pdhcg
