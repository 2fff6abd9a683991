// UP pair kernels for the AddU64 accumulation operator.
#include "pair_up.cuh"

namespace grgx {
void pair_up_u64(const PairUpParams<unsigned long long>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP8(AddU64)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
