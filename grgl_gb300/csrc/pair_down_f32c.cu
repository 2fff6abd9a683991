// DOWN pair kernels for compensated float32: rounded pattern rows by FastTwoSum, a single column's with their
// errors (PairTable).
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32c(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR_CASE(AddF32C, 1, 1)
    GRGX_PAIR_WIDE4(AddF32CPre<kF32Ordered>)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
