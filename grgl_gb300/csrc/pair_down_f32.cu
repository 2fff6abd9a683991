// DOWN pair kernels for the AddF32 accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR4(AddF32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
