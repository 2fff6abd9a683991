// Chains of small levels (chain.cuh), by accumulation operator.
#include "chain.cuh"

namespace grgx {
void launch_chain_u32(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN4(AddU32)
    throw std::runtime_error("unsupported sweep shape");
}
void launch_chain_xor(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN4(XorU32)
    throw std::runtime_error("unsupported sweep shape");
}
void launch_chain_u64(const ChainParams& p, int vw, int g, cudaStream_t s) {
    GRGX_CHAIN8(AddU64)
    throw std::runtime_error("unsupported sweep shape");
}

bool chain_supported() {
    constexpr int kMaxDev = 64;
    static std::atomic<int> known[kMaxDev];  // 0 unknown, 1 yes, 2 no
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDev) return false;
    int k = known[device].load(std::memory_order_relaxed);
    if (k == 0) {
        auto kernel = chain_kernel<AddU64, 2, 32>;
        int clusters = 0;
        const ChainLaunch c(nullptr);
        const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&clusters, kernel, &c.config) == cudaSuccess && clusters > 0;
        cudaGetLastError();
        k = ok ? 1 : 2;
        known[device].store(k, std::memory_order_relaxed);
    }
    return k == 1;
}

}  // namespace grgx
