// DOWN pair kernels for float64 as scaled float pairs (PackedF64ST).  The sweep sums runs of 32 edges in its float
// pairs, which short rows and few columns spread over several lanes, and folds them into doubles; here one lane
// has all of a row, and runs of 32 pattern rows folded into a float pair left more error than the sweep
// for few columns and for inputs of one sign.  Norm of the error against FP64 sums, 1e-15 of the norm, sweep / runs
// of 32 / of eight / of four; N(0,1) inputs, then their magnitudes:
//   200,000 samples and 3,000 variants (15 blocks),  K=2 3.1 / 3.8 / 3.3 / 2.6 and 1.43 / 2.74 / 1.78 / 1.10
//   200,000 and 10,000 (50),                         K=2 3.8 / - / 3.6 / 2.8 and 1.54 / - / 1.18 / 0.88
//   100,000 and 20,000 (100),                        K=2 4.2 / 5.6 / 3.5 / 2.8 and 1.40 / 2.47 / 0.94 / 0.77
//   200,000 and 250,000 (1,250),                     K=9 6.4 / 5.8 / 3.6 / - and 0.74 / 1.33 / 0.74 / -
// Milliseconds: 200,000 and 3,000 K=64 1.09 / 0.57 / 0.343 / 0.349; 100,000 and 20,000 K=64 1.51 / 0.52 / 0.49 / 0.51;
// 200,000 and 250,000 K=64 16.6 / 8.47 / 8.02 / 8.66, K=2 1.75 / 0.62 / 0.57 / 0.58.  The sums are read as float pairs,
// also between a launch's items: as doubles the conversions and additions alone took 0.23 of the 0.57 ms.
#include "pair_down.cuh"

namespace grgx {
void pair_down_f64s(const PairDownParams<DF>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s) {
    GRGX_PAIR8(AddF64ST)
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
