// solve_f32.cu -- FP32 (mixed-precision) instantiation of the pencil passes.
#include "solve_impl.cuh"

namespace gev {
GEV_SOLVE_INST(float)
int64_t fxy_partials(int N) { return N <= 128 ? N : (int64_t)(N / PASS_TX) * N; }
}  // namespace gev
