// UP pair kernels for the XorU32 accumulation operator.
#include "pair_up.cuh"

namespace grgx {
void pair_up_xor(const PairUpParams<uint32_t>& p, int vw, int g, cudaStream_t s) {
    GRGX_PAIR_UP4(XorU32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
