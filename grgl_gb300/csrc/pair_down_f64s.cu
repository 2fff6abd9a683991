// DOWN pair kernels for the AddF64S accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f64s(const PairDownParams<DF>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR8(AddF64SD)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
