// DOWN pair kernels for the XorU32 accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_xor(const PairDownParams<uint32_t>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR4(XorU32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
