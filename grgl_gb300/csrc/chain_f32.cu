// Chains of small levels (chain.cuh), by accumulation operator.
#include "chain.cuh"

namespace grgx {
void launch_chain_f32c(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN4(AddF32C)
    throw std::runtime_error("unsupported sweep shape");
}
void launch_chain_f32(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN4(AddF32)
    throw std::runtime_error("unsupported sweep shape");
}
}  // namespace grgx
