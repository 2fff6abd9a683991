// UP pair kernels for the AddU32 accumulation operator.
#include "pair_up.cuh"

namespace grgx {
void pair_up_u32(const PairUpParams<uint32_t>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP4(AddU32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
