// UP pair kernels for FP64 sums (grouped, as in pair_down_f32.cu).
#include "pair_up.cuh"

namespace grgx {
void pair_up_f64(const PairUpParams<double>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP8(AddF64G)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
