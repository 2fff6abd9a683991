// DOWN pair kernels for compensated float32 with a TwoSum per rounded pattern row (down_sums, pair_run.cu).
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32c1(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR_WIDE4(AddF32CPre<1>)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
