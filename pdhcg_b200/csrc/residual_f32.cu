// residual_f32.cu -- the residual kernels with FP32 iterates.
#include "residual_impl.cuh"

namespace pdhcg {

template void launch_residual<float>(const ResidualData<float> &, const ResidualParams &, int, bool, int, cudaStream_t);
template void launch_residual_psd<float>(const ResidualData<float> &, const ResidualParams &, const int *, int, int, int, int,
                                      cudaStream_t);

} // namespace pdhcg
