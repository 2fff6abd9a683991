// UP pair kernels for plain float32 (grouped, as in pair_down_f32.cu).
#include "pair_up.cuh"

namespace grgx {
void pair_up_f32(const PairUpParams<float>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP4(AddF32G)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
