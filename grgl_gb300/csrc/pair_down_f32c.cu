// DOWN pair kernels for the AddF32C accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32c(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR4(AddF32C)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
