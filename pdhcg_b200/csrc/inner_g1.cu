// inner_g1.cu -- inner BB solve, 1 lane per row of Q.
#include "inner_impl.cuh"

namespace pdhcg {
PDHCG_INNER(1)
} // namespace pdhcg
