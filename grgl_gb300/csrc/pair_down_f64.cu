// DOWN pair kernels for the AddF64 accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f64(const PairDownParams<double>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR8(AddF64)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
