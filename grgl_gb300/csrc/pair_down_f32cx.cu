// DOWN pair kernels for compensated float32 over pattern rows that keep their error, two columns a lane.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32cx(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR_CASE(AddF32CX, 2, 1)
    GRGX_PAIR_CASE(AddF32CX, 2, 2)
    GRGX_PAIR_CASE(AddF32CX, 2, 4)
    GRGX_PAIR_CASE(AddF32CX, 2, 8)
    GRGX_PAIR_CASE(AddF32CX, 2, 16)
    GRGX_PAIR_CASE(AddF32CX, 2, 32)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
