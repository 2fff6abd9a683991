// DOWN pair kernels for the AddU64 accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_u64(const PairDownParams<unsigned long long>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR8(AddU64)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
