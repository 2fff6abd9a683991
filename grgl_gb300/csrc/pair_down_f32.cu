// DOWN pair kernels for plain float32 (GroupedAcc).  The sweep spreads a narrow row's edges over up to 32 lanes and
// merges their sums; here one lane has all of a row, and adding its pattern rows one after the other left up to
// three times the sweep's error in few columns (and a third of it in many).  Norm of the error, 1e-8 of the norm, sweep /
// one by one / grouped (eight rows as a tree, eight groups of four to a run); N(0,1) inputs, then their magnitudes:
//   100,000 samples and 20,000 variants, K=2 11.9 / 21.8 / 11.3 and 4.3 / 15.7 / 4.9, K=64 20 / 20 / 10 and 12 / 16 / 5
//   200,000 and 250,000, K=2 19 / 21 / 12 and 3.8 / 6.9 / 5.6, K=64 65 / 25 / 11 and 35 / 8 / 5
// UP K=9 on 100,000 and 20,000 13.9 / 20.4 / 11.3.  FP64 sums (pair_down_f64.cu), 1e-17 of the norm: K=2 on 100,000 and
// 20,000 8.9 / 34 / 10.6, on 200,000 and 250,000 31 / 45 / 17, K=18 127 / 62 / 15.
// Microseconds on 200,000 and 250,000, one by one / grouped: K=5 784 / 789, K=32 1809 / 1794; UP K=5 1195 / 1186, K=20
// 1837 / 1997; FP64 K=2 1105 / 1133, K=20 10,720 / 11,010, UP K=2 2047 / 2333 (2,360, 31,400 and 2,500 in the sweep).  Beside
// float pairs, whose kernels have no registers for runs, the FP64 path has trees of four alone.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f32(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR4(AddF32G)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
