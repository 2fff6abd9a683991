// UP pair kernels for compensated float32.  A pattern row is rounded to float32, which takes the
// place of the pre-sums a height-0 edge passes in the sweep: its lists are summed by FastTwoSum
// (kF32Ordered), and the nodes' lists over table rows by TwoSum.  A pre-sum of two rows before a TwoSum in the
// patterns' lists has as many operations and 10% more error (N=50,000, M=50,000, N(0,1) inputs, 1e-8 of the
// norm: K=2 5.4 against 4.9, K=64 5.6 and 4.9, the sweep 5.9 and 6.4; standardized 6.4, 5.9 and 6.4), but frees the rows'
// registers sooner.  With four lanes to a row that counts: K=16 on N=200,000, M=250,000 1.42 ms against 1.47, N=1,000,000,
// M=50,000 K=64 (tiles of four lanes) 5.26 against 5.97; elsewhere FastTwoSum is as fast or faster (K=4 1.32 and 1.18,
// K=64 4.39 and 4.40, N=400,000, M=100,000 K=256 14.7 and 14.2).  Four lanes keep the pre-sum, which is below the
// sweep's error for the nine columns or more that they have (K=9 plain 5.5 against 6.4, standardized 6.3 and 6.9).
#include "pair_up.cuh"

namespace grgx {
void pair_up_f32c(const PairUpParams<float>& p, int vw, int g, cudaStream_t s) {
    if (p.second) {
        GRGX_PAIR_UP4(AddF32CPre<1>)
    } else {
        GRGX_PAIR_UP_CASE(AddF32CPre<2>, 4, 4)
        GRGX_PAIR_UP4_BUT4(AddF32CPre<kF32Ordered>)
    }
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
