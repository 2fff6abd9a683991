// UP pair kernels for the AddF32 accumulation operator.
#include "pair_up.cuh"

namespace grgx {
void pair_up_f32(const PairUpParams<float>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP4(AddF32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
