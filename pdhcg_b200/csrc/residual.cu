// residual.cu -- the residual kernel (residual.cuh) and its launcher.
#include "launch.cuh"

namespace pdhcg {

template <typename VT>
void launch_residual(const ResidualData<VT> &D, const ResidualParams &P, int S, bool fixed, int blocks, cudaStream_t s)
{
    if (fixed) // one slot class for problems with fixed cone slots
        residual_kernel<8, VT, true><<<blocks, TPB, 0, s>>>(D, P);
    else
        dispatch_s(S, [&](auto SC) { residual_kernel<SC.value, VT, false><<<blocks, TPB, 0, s>>>(D, P); });
}

template void launch_residual<double>(const ResidualData<double> &, const ResidualParams &, int, bool, int,
                                      cudaStream_t);
template void launch_residual<float>(const ResidualData<float> &, const ResidualParams &, int, bool, int, cudaStream_t);

} // namespace pdhcg
