// Host-side launch entry points of the device kernels (internal to libgrgx).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "sweep.cuh"

namespace grgx {

// SM count of the current device (looked up once per device, matmul.cu).
int sm_count();

// Storage/accumulation kinds (see ops.cuh).
enum class Kind { U32, U64, F64, F32C, F32, XOR, F64S };

// One level (or seed pass) of the sweep; VW elements per lane, G lanes per row, `variant` 0 for
// the default depth or 1 for the deep variant (float32, compensated float32, int32 and
// float-pair float64 storage only).
void launch_sweep_u32(const SweepParams<uint32_t>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_xor(const SweepParams<uint32_t>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_u64(const SweepParams<unsigned long long>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_f64(const SweepParams<double>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_f32c(const SweepParams<float>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_f32(const SweepParams<float>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);
void launch_sweep_f64s(const SweepParams<DF>& p, int vw, int g, int variant, dim3 grid,
                      int sms, cudaStream_t s);

// Chains of small levels (chain.cuh): up to kChainMost levels in one launch of one cluster.
constexpr int kChainMost = 24, kChainBlocks = 16, kChainThreads = 1024;
struct ChainLevel {
    const unsigned* off;   // first edge of each row (rows + 1), relative to adj
    const uint32_t* adj;
    const int* nodes;      // destination of each row
    const void* src;       // rows gathered from
    unsigned rows;
    int split, rmw;
};
struct ChainParams {
    ChainLevel level[kChainMost];
    int count, tiles;      // tiles: of G x VW columns
    void* vals;
    long long stride;
    void* state;           // as SweepParams::state, mode 2
    long long state_base;
    const int* gate;       // as SweepParams::gate
};
bool chain_supported();  // the device takes a cluster of that size
void launch_chain_u32(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_xor(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_u64(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_f64(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_f32c(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_f32(const ChainParams& p, int vw, int g, cudaStream_t s);
void launch_chain_f64s(const ChainParams& p, int vw, int g, cudaStream_t s);

// The pair form's ids are padded by at least this many height-0 rows: no warp takes more at a time.
constexpr int kPairTile = 128;

// DOWN in pair form (pair_down.cuh): one launch over `items` shares of the blocks (groups of four,
// group_begin .. group_end) x `tiles` row tiles.
template <typename S> struct PairDownParams {
    const uint2* ids;    // four 16-bit pattern numbers per (row tile of 32, group, row)
    const uint4* base;   // first pattern of each block, by groups of four
    void* table;         // pattern rows, from pattern `base0` on
    S* vals;             // node values (the height-0 rows first)
    void* parts;         // one sum per (item, row, column), or null: rows are written at once
    unsigned* work;      // per column tile: next item (zeroed before the launch)
    long long rows, stride, groups;
    unsigned base0, tiles, items;
    int group_begin, group_end, groups_per_item, part_begin;
    int long_runs;       // float pairs: runs of eight rows (0: of four)
    const int* gate;  // as SweepParams::gate
};
// What a pair_down_* call does, and what its kShape step answers.
struct PairDownCall {
    enum Step { kShape, kTable, kGather, kFinish } step = kShape;
    int rows_per_warp = 0, resident_warps = 0;  // kShape
    size_t part_bytes = 0, table_bytes = 0;     // per element of a sum and of a pattern row
    const uint2* nodes = nullptr;  // kTable: the patterns' parents
    long long count = 0;
    int parts = 0;      // kFinish: sums per row
    bool onto = false;  // kFinish: onto the node values (else into the first sum)
};
void pair_down_u32(const PairDownParams<uint32_t>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_xor(const PairDownParams<uint32_t>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_u64(const PairDownParams<unsigned long long>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f64(const PairDownParams<double>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f32c1(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f32cx(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f32c(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f32(const PairDownParams<float>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);
void pair_down_f64s(const PairDownParams<DF>& p, PairDownCall& c, int vw, int g, int sms, cudaStream_t s);

// UP in pair form (pair_up.cuh): sums over `count` lists of source rows.
struct PairList {
    long long e0;  // first id
    int len;
    int out;       // destination row; ~row for a row of the table
};
template <typename S> struct PairUpParams {
    const PairList* lists;
    long long count;
    const uint32_t* adj;
    const S* src;
    S* table;      // pattern rows
    S* dst;        // the nodes' rows of sums (added onto when rmw), or
    int rmw;
    void* state;   // when set, accumulators (Op::A)
    int second;    // sums for nodes (0: pattern rows)
    long long stride;
    long long src_stride, tile_step;  // elements from a source row to the next, from a column tile to the next
    const int* gate;  // as SweepParams::gate
};
void pair_up_u32(const PairUpParams<uint32_t>& p, int vw, int g, cudaStream_t s);
void pair_up_xor(const PairUpParams<uint32_t>& p, int vw, int g, cudaStream_t s);
void pair_up_u64(const PairUpParams<unsigned long long>& p, int vw, int g, cudaStream_t s);
void pair_up_f64(const PairUpParams<double>& p, int vw, int g, cudaStream_t s);
void pair_up_f32c(const PairUpParams<float>& p, int vw, int g, cudaStream_t s);
void pair_up_f32(const PairUpParams<float>& p, int vw, int g, cudaStream_t s);
void pair_up_f64s(const PairUpParams<DF>& p, int vw, int g, cudaStream_t s);

// Column-map modes of the transposing loads/stores.
enum MapMode { MAP_IDENT = 0, MAP_DIV = 1, MAP_TABLE = 2, MAP_FOLD = 3 };

// Loads and stores of few columns take a thread per row instead of tiles of 32 columns, which do 32 columns'
// work for them.  Whole products, tiles against threads per row, in us: 200,000 samples and 250,000
// mutations, int32 UP K=1 403 / 381, K=8 1199 / 1181, K=20 1853 / 1833, float64 DOWN K=1 490 / 436, K=20 3010 /
// 3000; 60,000 and 100,000, float64 UP K=8 365 / 349, K=20 601 / 596.  With fewer rows the threads are too
// few to hide a long row: 20,000 and 50,000, float64 DOWN K=4 101 / 95, K=20 204 / 209; 1,000 and 10,000, K=4
// 63 / 61, K=8 63 / 65, int32 DOWN K=8 45 / 44, K=20 50 / 50.
inline bool narrow_io(long long K, long long rows, size_t size) {
    return K * static_cast<long long>(size) <= 48 || (K <= 20 && rows >= 60000);
}
// Calls f with the elements per vector of a row of `stride` elements of Size bytes (choose_layout).
template <size_t Size, typename F> void narrow_vec(long long stride, F&& f) {
    if (stride == 1) {
        f(std::integral_constant<int, 1>{});
    } else if constexpr (Size == 4) {
        if (stride == 2) f(std::integral_constant<int, 2>{});
        else f(std::integral_constant<int, 4>{});
    } else {
        f(std::integral_constant<int, 2>{});
    }
}

// dst[i*stride + k] (=, or += when add) IO->S(src[k*ld + col(i)]) for i < R, k < K; columns
// K..stride-1 are zeroed when assigning.  col(i) = i, i/div, or tab[i].
void launch_load_rows(int dtype, const void* src, long long K, long long ld, long long R, int mode, long long div,
                      const uint32_t* tab, void* dst, long long stride, int add, cudaStream_t s);

// out[k*ld + c] (=, or += when add) S->IO(vals[map(c)]) for c < C, k < K; map(c) = c, tab[c]
// (INVALID -> 0), or the sum of rows c*fold .. c*fold+fold-1.
void launch_store_cols(int dtype, const void* vals, long long stride, long long K, long long C, int mode,
                       long long fold, const uint32_t* tab, void* out, long long ld, int add, cudaStream_t s);

// Node-value initialisation: VECTOR (vals[v][k] = init[k]) and XTX (vals[v][k] = xtx[v]).
void launch_init_vector(int dtype, const void* init, long long K, long long n, void* vals, long long stride,
                        cudaStream_t s);
void launch_init_xtx(int dtype, const uint32_t* xtx, long long K, long long n, void* vals, long long stride,
                     cudaStream_t s);

// ---- float64 as scaled float pairs (AddF64S) ----------------------------------------------
// rowmax[k] = max over finite |x| of row k, as IEEE bits (0 for an all-zero row); callers
// fill it first (0, or a floor such as the largest XTX init value) and may fold several
// matrices into it.  Row k is scaled by 2^(60 - e_k), e_k the exponent of rowmax[k], so the
// row's largest value sits in [2^60, 2^61) and values down to 2^-126 of float range (186
// binades below the maximum) keep full precision.  When gate[0] != 0 the same launches move plain
// doubles instead (the call takes the FP64 path).
void launch_fill_u64(unsigned long long* p, long long n, unsigned long long v, cudaStream_t s);
// Also folds the smallest nonzero finite magnitude into rowmin[k] (filled with ~0 first).
void launch_rowmax(const double* src, long long K, long long ld, long long cols, unsigned long long* rowmax,
                   unsigned long long* rowmin, cudaStream_t s);
// gate[0] = 1 when some row spans more binades than the float-pair path holds, or holds an inf
// or a nan (the call then runs on the FP64 pipe), else 0.
void launch_decide_f64_path(const unsigned long long* rowmax, const unsigned long long* rowmin, long long K, int* gate,
                            cudaStream_t s);
void launch_load_rows_df(const double* src, long long K, long long ld, long long R, int mode, long long div,
                         const uint32_t* tab, void* dst, long long stride, int add,
                         const unsigned long long* rowmax, cudaStream_t s, const int* gate);
void launch_store_cols_df(const void* vals, long long stride, long long K, long long C, int mode, long long fold,
                          const uint32_t* tab, double* out, long long ld, int add,
                          const unsigned long long* rowmax, cudaStream_t s, const int* gate);
void launch_init_vector_df(const double* init, long long K, long long n, void* vals, long long stride,
                           const unsigned long long* rowmax, cudaStream_t s, const int* gate);
void launch_init_xtx_df(const uint32_t* xtx, long long K, long long n, void* vals, long long stride,
                        const unsigned long long* rowmax, cudaStream_t s, const int* gate);

}  // namespace grgx
