// UP pair kernels for float64 as scaled float pairs.  Table rows are many times larger than the
// height-0 values behind them, and so are the errors of adding them up in runs: the nodes' lists add
// them with normalised pairs throughout.
#include "pair_up.cuh"

namespace grgx {
void pair_up_f64s(const PairUpParams<DF>& p, int vw, int g, cudaStream_t s) {
    if (p.second) {
        GRGX_PAIR_UP8(AddF64SN)
    } else {
        GRGX_PAIR_UP8(AddF64SD)
    }
    throw std::runtime_error("unsupported pair shape");
}
}  // namespace grgx
