// UP pair kernels for the AddF64 accumulation operator.
#include "pair_up.cuh"

namespace grgx {
void pair_up_f64(const PairUpParams<double>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP8(AddF64)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
