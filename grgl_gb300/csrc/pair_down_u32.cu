// DOWN pair kernels for the AddU32 accumulation operator.
#include "pair_down.cuh"

namespace grgx {
void pair_down_u32(const PairDownParams<uint32_t>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR4(AddU32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
