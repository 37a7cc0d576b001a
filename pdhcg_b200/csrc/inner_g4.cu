// inner_g4.cu -- inner BB solve, 4 lanes per row of Q.
#include "inner_impl.cuh"

namespace pdhcg {
PDHCG_INNER(4)
} // namespace pdhcg
