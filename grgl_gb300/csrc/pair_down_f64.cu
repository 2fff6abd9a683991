// DOWN pair kernels for FP64 sums (grouped, as in pair_down_f32.cu).
#include "pair_down.cuh"

namespace grgx {
void pair_down_f64(const PairDownParams<double>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR8(AddF64G)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
