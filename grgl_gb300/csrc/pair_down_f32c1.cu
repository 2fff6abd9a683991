// DOWN pair kernels for compensated float32 without a pre-sum of pattern rows (down_sums, pair_run.cu).
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32c1(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR_CASE(AddF32CPre<1>, 2, 1)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 1)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 2)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 4)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 8)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 16)
    GRGX_PAIR_CASE(AddF32CPre<1>, 4, 32)
    GRGX_PAIR_ODD(AddF32CPre<1>, 4)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
