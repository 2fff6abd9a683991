// Chains of small levels (chain.cuh), by accumulation operator.
#include "chain.cuh"

namespace grgx {
void launch_chain_f64s(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN8(AddF64S)
    throw std::runtime_error("unsupported sweep shape");
}
void launch_chain_f64(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN8(AddF64)
    throw std::runtime_error("unsupported sweep shape");
}
}  // namespace grgx
