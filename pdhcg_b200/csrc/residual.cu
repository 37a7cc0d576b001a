// residual.cu -- the residual kernels with FP64 iterates.
#include "residual_impl.cuh"

namespace pdhcg {

bool residual_psd_fits(int order) { return residual_psd_smem(order) <= RESIDUAL_PSD_SMEM; }

template void launch_residual<double>(const ResidualData<double> &, const ResidualParams &, int, bool, int, cudaStream_t);
template void launch_residual_psd<double>(const ResidualData<double> &, const ResidualParams &, const int *, int, int, int, int,
                                      cudaStream_t);

} // namespace pdhcg
