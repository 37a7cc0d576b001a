// inner_g32.cu -- inner BB solve, 32 lanes per row of Q.
#include "inner_impl.cuh"

namespace pdhcg {
PDHCG_INNER(32)
} // namespace pdhcg
