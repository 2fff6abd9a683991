// UP pair kernels for compensated float32.  A pattern row is rounded to float32, which takes the
// place of one of the two pre-sum levels a height-0 edge passes in the sweep: its lists pre-sum two
// rows, and the nodes' lists over table rows none.
#include "pair_up.cuh"

namespace grgx {
void pair_up_f32c(const PairUpParams<float>& p, int vw, int g, cudaStream_t s) {
    if (p.second) {
        GRGX_PAIR_UP4(AddF32CPre<1>)
    } else {
        GRGX_PAIR_UP4(AddF32CPre<2>)
    }
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
