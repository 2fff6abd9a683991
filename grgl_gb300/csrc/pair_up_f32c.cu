// UP pair kernels for compensated float32.  A pattern row is rounded to float32, which takes the
// place of the pre-sums a height-0 edge passes in the sweep: its lists are summed by FastTwoSum
// (kF32Ordered), and the nodes' lists over table rows by TwoSum.  A pre-sum of two rows in the patterns'
// lists took as long and left 10% more error (N=50,000, M=50,000, N(0,1) inputs, 1e-8 of the norm: K=6 5.6 against
// 5.0, K=64 5.6 and 4.9, the sweep 6.3 and 6.4; standardized K=6 6.3, 5.8 and 6.7).
#include "pair_up.cuh"

namespace grgx {
void pair_up_f32c(const PairUpParams<float>& p, int vw, int g, cudaStream_t s) {
    if (p.second) {
        GRGX_PAIR_UP4(AddF32CPre<1>)
    } else {
        GRGX_PAIR_UP4(AddF32CPre<kF32Ordered>)
    }
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
