// Device-resident plan and launch helpers shared by the matmul entry points (internal).
#pragma once
#include <cuda_runtime.h>

#include <map>
#include <string>
#include <vector>

#include "grgx_internal.h"
#include "launch.h"
#include "pair_plan.h"

namespace grgx {

#define GRGX_CUDA(call)                                                                               \
    do {                                                                                             \
        cudaError_t err__ = (call);                                                                  \
        if (err__ != cudaSuccess) {                                                                  \
            const int code__ = (err__ == cudaErrorMemoryAllocation) ? GRGX_ERR_OUT_OF_MEMORY         \
                                                                    : GRGX_ERR_CUDA;                 \
            throw ::grgx::Error(code__, std::string(#call) + ": " + cudaGetErrorString(err__));       \
        }                                                                                            \
    } while (0)

struct DevCSR {
    uint32_t* adj = nullptr;  // 32-bit ids, or 16-bit block-relative ids when id16
    bool id16 = false;
    // id16: per level (= split block), the block's first source id and its number of source ids
    std::vector<long long> level_base, level_src_rows;
    int* rows = nullptr;
    ChunkDev* chunks = nullptr;
    HeavyDev* heavy = nullptr;
    std::vector<int32_t> lb, le;
    std::vector<long long> level_rows, level_edges;  // per level, for the launch-shape table
    // per level of short rows, or small enough for a chain: its rows' first edges, relative to
    // level_e0 (else null)
    std::vector<unsigned*> level_short;
    // ... and whether short_rows_kernel takes it (else the offsets serve chains only)
    std::vector<char> level_alone;
    std::vector<long long> level_r0, level_e0;
    std::vector<int> level_most;  // its longest row
    long long n_heavy = 0, n_pieces = 0, n_edges = 0, n_rows = 0;
};

// A share of one split block's lists (staged.cu): parts `part` of `parts`.
struct StagedPart {
    long long src;  // the block's first source id
    int rows;       // its source ids
    int list0, list1;
    int part, parts;
};
// The lists of a split copy for single-column products.
struct StagedLists {
    StagedPart* parts = nullptr;
    unsigned nparts = 0;
    PairList* lists = nullptr;              // out = slot
    unsigned* slot0 = nullptr;              // first slot of each row (+ the end)
    int* nodes = nullptr;
    const unsigned short* adj = nullptr;
    long long rows = 0, slots = 0;
};

struct DevicePlan {
    int device = -1;
    DevCSR up, down, seed, miss;
    // up / down (and below up0b, up_int, down0b) on the fine chunking: the same adjacency and
    // rows, kFineChunkFactor times the chunks per level (sweep_csrs picks them for wide rows)
    DevCSR up_f, down_f;
    // UP in split form (empty when the height-0 nodes make fewer than two blocks):
    //   up0b    the edges to height-0 children, cut by blocks of `split_block` height-0 ids;
    //           level j = block j, rows = every node with children in the block
    //   up_int  the edges to children of height >= 1, one level per UP level (same order)
    //   fin     per UP level, the nodes without such children (finished from their state alone),
    //           concatenated; fin_begin[j] .. fin_begin[j+1] for level j
    // Built on the first call that runs UP in split form (use_up_split), from the UP row offsets
    // and level boundaries kept here.
    DevCSR up0b, up_int, up0b_f, up_int_f;
    int* fin = nullptr;
    std::vector<long long> fin_begin;
    bool up_int_built = false;                 // (up_int, fin: also used by the pair form)
    long long split_block = 0, split_src = 0;  // split_src = height-0 ids = first UP row's node id
    bool split_built = false;
    std::map<std::pair<int, long long>, bool> split_choice;  // (storage kind, stride) -> measured choice
    // DOWN in split form (empty when the parents of height-0 rows make fewer than two blocks):
    //   down0b  the edges of the height-0 DOWN rows, cut by blocks of `split_block` parent ids
    //           starting at split_src (parents all have height >= 1); level j = block j, rows =
    //           every height-0 row with parents in the block; 16-bit block-relative ids
    //   fin_down the height-0 DOWN rows, finished from their state after the block passes
    // Built on the first call that runs DOWN in split form (use_down_split).
    DevCSR down0b, down0b_f;
    StagedLists up_staged, down_staged;  // built with the split copies
    int* fin_down = nullptr;
    long long n_fin_down = 0;
    bool down_split_built = false;
    std::map<std::pair<int, long long>, bool> down_split_choice;
    std::map<std::pair<int, long long>, bool> up_pair_choice, down_pair_choice;  // pair form or not, measured
    PairPlan pair;                       // pair form of the height-0 edges, on first use (use_pair_form)
    std::vector<int64_t> down_off;       // DOWN row offsets (host copy)
    long long down_h0_row = 0;           // first DOWN row of height 0
    std::vector<int64_t> up_off;         // UP row offsets (host copy)
    std::vector<uint64_t> level_begin;   // node-id range of each height
    uint32_t* mut_new = nullptr;
    uint32_t* miss_new = nullptr;
    uint32_t* old2new = nullptr;
    uint32_t* new2old = nullptr;
    uint32_t* xtx_new = nullptr;
    uint64_t bytes = 0;
    uint64_t num_levels = 0;
    bool has_coals = false;
    bool has_miss = false;
    double xtx_max = 0.0;  // largest XTX init value (2 * coalescences)
    double* freq = nullptr;       // allele frequency per mutation (standardized products)
    double* inv_sigma = nullptr;  // 1/sqrt(p(1-p)) per mutation, 0 where p(1-p) == 0
    std::vector<void*> allocs;
};

struct Layout {
    Kind kind;
    int ssize;     // storage bytes per element
    int asize;     // accumulator bytes per element (heavy partials)
    long long stride;
    int vw, g, ntiles;
};

// Element layout of one call: storage kind, row stride and the default (VW, G) sweep shape.
Layout choose_layout(int dtype, long long K, bool plainF32, bool nativeF64);

// Launch shape of one level: G lanes per row, the column tiles that G leaves (the K-tile
// count), and the prefetch-depth variant (0 default, 1 deep).
struct LevelShape {
    int g = 1;
    int ntiles = 1;
    int variant = 0;
};
LevelShape default_shape(const Layout& L);
// The shape a level runs with: the autotuner's entry for (storage kind, row stride, the level's
// width and mean degree) when there is one, else the default.
LevelShape level_shape(const Layout& L, const DevCSR& c, size_t level);
// Column tiles of the widest shape the autotuner may pick for L: the stride of the per-launch
// work counters and of the heavy-row tickets.
int max_tiles(const Layout& L);

// The sweep CSRs a call with layout L runs on: rows of 32 bytes or more (K >= 8 four-byte or
// K >= 4 eight-byte values) take the fine chunking, narrower rows -- whose chunks cost little
// each, so that more of them only adds per-chunk work (the staged single-column passes lose
// 10-20%) -- the coarse one.  The split copies' members are empty until they are built.
// Device memory of a plan (cudaMalloc).  set_plan_alloc (tests): `pass` more allocations are made, `refuse`
// after them fail as out of memory (pass -1: none fail); returns how many have failed since the last call.
void* plan_alloc(size_t bytes);
long long set_plan_alloc(long long pass, long long refuse);
// What a build adds to a plan is handed over when it has succeeded: freed again unless kept.
class PlanAddition {
  public:
    explicit PlanAddition(DevicePlan& d) : d_(d), count_(d.allocs.size()), bytes_(d.bytes) {}
    ~PlanAddition() {
        if (kept_) return;
        for (size_t i = count_; i < d_.allocs.size(); i++) cudaFree(d_.allocs[i]);
        d_.allocs.resize(count_);
        d_.bytes = bytes_;
    }
    void keep() { kept_ = true; }
    PlanAddition(const PlanAddition&) = delete;
    PlanAddition& operator=(const PlanAddition&) = delete;

  private:
    DevicePlan& d_;
    size_t count_;
    uint64_t bytes_;
    bool kept_ = false;
};

struct SweepCSRs {
    const DevCSR* up;
    const DevCSR* down;
    const DevCSR* up0b;
    const DevCSR* up_int;
    const DevCSR* down0b;
};
bool fine_chunks(const Layout& L);
SweepCSRs sweep_csrs(const DevicePlan* dp, const Layout& L);
// Uploads rows, chunks and heavy rows of P; `adj` (E ids) is on the device already.  blockBase and
// blockRows set: 16-bit ids, level j = the block of blockRows[j] source ids from blockBase[j] on.
DevCSR upload_pull(DevicePlan& d, const PullCSR& P, void* adj, long long E,
                   const std::vector<long long>* blockBase = nullptr, const std::vector<long long>* blockRows = nullptr);
// Finds the levels of `r` whose rows are short (rows' offsets `off`, chunks of `c`) and uploads their
// offsets.
void mark_short_levels(DevicePlan& d, DevCSR& r, const PullCSR& c, const std::vector<int64_t>& off);
// `coarse` with the chunks, heavy rows and level ranges of `fine` (uploaded; the adjacency and
// rows are shared).
DevCSR fine_view(DevicePlan& d, const DevCSR& coarse, const PullCSR& fine);

// Launches one level of a CSR (a no-op when the level has no chunks); `work` points at
// `tileStride` (0: L.ntiles) zeroed counters owned by this launch, and the heavy-row tickets
// are `tileStride` apart.  `shape` null: the default shape.  Returns the kernels launched.
// `state` set: each node's Op::A accumulator lives at state + (node - stateBase) rows; with
// stateMode 1 a row's sum is merged into it (nothing written), with 2 the node value is written
// from the accumulator merged with the row's sum.
int launch_level(const Layout& L, const DevCSR& c, size_t level, const void* src, void* dst, int rmw,
                 void* partials, unsigned* tickets, unsigned* work, cudaStream_t s, const int* gate = nullptr,
                 const LevelShape* shape = nullptr, int tileStride = 0, void* state = nullptr,
                 long long stateBase = 0, int stateMode = 1);

// Levels first .. last-1 of a CSR, launched one by one or, where consecutive ones are short and small,
// as chains (chain.cuh).  `seed` set: its level 0 (gathering from seedSrc, seedRmw) goes first.
// `tickets` and `work` as for launch_level, level lvl's counters at work + lvl * tileStride (the
// seed's own: seedTickets, seedWork).
struct LevelRun {
    const DevCSR* csr = nullptr;
    size_t first = 0, last = 0;
    int rmw = 0;
    unsigned *tickets = nullptr, *work = nullptr;
    const DevCSR* seed = nullptr;
    const void* seedSrc = nullptr;
    int seedRmw = 0;
    unsigned *seedTickets = nullptr, *seedWork = nullptr;
    void* state = nullptr;  // mode 2
    long long stateBase = 0;
};
int launch_levels(const Layout& L, const LevelRun& run, void* vals, void* partials, int tileStride, cudaStream_t s,
                  const int* gate);

// UP in split form (up_split.cu): writes vals[node] from its accumulator state (added onto the
// value when rmw) for the `count` nodes listed at `nodes`.
void launch_state_finish(Kind kind, const void* state, void* vals, const int* nodes, long long count,
                         long long stateBase, long long stride, int rmw, cudaStream_t s, const int* gate);
// Height-0 row bytes (height-0 ids x stride x element size) above which UP runs in split form,
// and the block of height-0 ids each split pass covers; both adjustable for tests.
constexpr unsigned long long kDefaultSplitThreshold = 64ull << 20;
uint64_t split_threshold_bytes();
long long split_block_size();
// Whether a call with layout L runs UP in split form: the choice grgx_autotune measured for
// (storage kind, stride) on this graph, else whether the height-0 rows exceed the threshold.
// Builds the split copy on first use.
bool use_up_split(grgx_graph* g, DevicePlan* dp, const Layout& L);
bool up_split_possible(const DevicePlan* dp);
void ensure_up_split(grgx_graph* g, DevicePlan* dp);
void set_up_split_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool split);
// The same for DOWN: the height-0 level in parent blocks.  Without a measured choice a call runs
// DOWN in split form when its block passes run staged (staged_layout); UP likewise, or when the
// height-0 rows exceed the threshold.
bool use_down_split(grgx_graph* g, DevicePlan* dp, const Layout& L);
bool down_split_possible(const DevicePlan* dp);
void ensure_down_split(grgx_graph* g, DevicePlan* dp);
void set_down_split_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool split);
// Whether layout L runs its split form staged: a single 4-byte column (K = 1 for the 4-byte dtypes,
// bool up to 32 columns), whose source blocks fit in shared memory (staged.cu); on by default,
// switchable for tests.
constexpr long long kStagedRows = 32768;
bool staged_enabled();
void set_staged(bool on);
bool staged_layout(const Layout& L);
// The rows' sums over their height-0 children (UP) or parents (DOWN) on T's lists: into `state` (from
// node stateBase on) or onto / into vals; `sums` holds T.slots accumulators.
int launch_staged(Kind kind, const StagedLists& T, void* vals, void* sums, void* state, long long stateBase, int rmw,
                  cudaStream_t s);
// The lists of a split copy: per row (R) and block (nb) its segment bounds `seg` and place `start`.
void build_staged(DevicePlan& d, StagedLists& T, const std::vector<uint32_t>& seg, const std::vector<long long>& start,
                  long long R, int nb, const std::vector<long long>& base, const std::vector<long long>& srcRows,
                  const std::vector<int>& nodeOf, const unsigned short* adj);
// DOWN split form: 0 chosen as above, 1 always (where possible), 2 never (tests).
void set_down_split_mode(int mode);
bool down_split_forced();

// Whether a call with layout L on stream s runs in pair form (pair_plan.h); builds the form on the first call
// that may use it, unless s is being captured into a CUDA graph.  set_pair_mode: 0 by the rules, 1 wherever possible, 2 never (tests).
bool use_pair_form(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, cudaStream_t s);
// Scratch the pair form of a call on this thread may take beyond what the other forms need; a
// server's worker lowers it to what its batch has reserved (PairScratchScope).
size_t pair_scratch_limit();
void set_pair_mode(int mode);
// What grgx_autotune measured for L's (storage kind, stride) on this graph; clear_pair_choice: the rules again.
void set_pair_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, bool pair);
void clear_pair_choice(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down);
void set_pair_rows(long long most);  // UP table rows from which that direction keeps the other forms (tests)
// out: height-0 nodes, blocks, patterns, height-0 edges of a direction in pair form (zeros: not in use).
void pair_counts(grgx_graph* g, bool down, uint64_t out[4]);
// Where the analysis that calls read without the graph's lock is held (null: none; tests).
const void* pair_analysis(grgx_graph* g);
// The launches of a DOWN call in pair form, sized for layout L: a table of pattern rows per range
// of blocks, and per range the sums of its items.  With several ranges the first sum carries what
// the ranges before added up.
struct PairDownRun {
    struct Range {
        int g0, g1;  // groups of four blocks
        long long pat0, count;
        int items, groups_per_item;
    };
    std::vector<Range> ranges;
    int tiles = 1;  // column tiles: counters per range
    int slots = 0;  // sums per row held at a time (0: the only item writes its rows)
    size_t table_bytes = 0, part_bytes = 0;
};
// `limit`: most bytes of scratch the table and the sums may take; no ranges where that is too little.
PairDownRun pair_down_run(const Layout& L, const DevicePlan* dp, size_t limit);
// Adds the height-0 rows' sums onto vals; `work` holds run.tiles zeroed counters per range.
// Returns the kernels launched.
int launch_pair_down(const Layout& L, const DevicePlan* dp, const PairDownRun& run, void* vals, void* table, void* parts,
                     unsigned* work, cudaStream_t s, const int* gate);

// The launches of an UP call in pair form: ranges of segments, with a table of pattern rows at a
// time.
struct PairUpRun {
    struct Range {
        size_t s0, s1;  // segments
    };
    std::vector<Range> ranges;
    size_t table_bytes = 0;
    size_t source_bytes = 0;  // behind the table: the height-0 rows by column tiles, or none
    size_t bytes() const { return table_bytes + source_bytes; }
};
PairUpRun pair_up_run(const Layout& L, const DevicePlan* dp, size_t limit);
// A call's pair form within this thread's scratch limit: its direction's launches, without ranges where it
// takes another form.
struct PairRuns {
    PairUpRun up;
    PairDownRun down;
    // UP: compensated float32 keeps the sums as pairs until a node's other children are added; every other
    // kind adds them onto the node's value
    size_t up_state_bytes = 0;
};
PairRuns pair_runs(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, cudaStream_t s);
// Writes every node's sum over its height-0 children to vals (onto it when rmw), or leaves it in
// `state` where one is given.
int launch_pair_up(const Layout& L, const DevicePlan* dp, const PairUpRun& run, void* vals, void* table, void* state,
                   int rmw, cudaStream_t s, const int* gate);
// Builds the UP edges to children of height >= 1 (up_int and the finish lists), once: `low` = each
// UP row's children of height 0.  The caller holds the graph's lock.
void build_up_internal(DevicePlan& d, const std::vector<unsigned>& low);
std::vector<unsigned> count_low_children(DevicePlan& d);

// Resolves (once per device, with `device` current) the address of grgx_matmul_noalloc's
// static scratch, which loads its module and so reserves the array on the device.
void noalloc_prepare_device(int device);

// Builds (once) and returns the graph's plan on the current device.
DevicePlan* ensure_device_plan(grgx_graph* g);

// The library's own stream-ordered memory pool on `device` (created on first use).
cudaMemPool_t library_pool(int device);
// Bytes of the library pool on `device` handed out to calls now, and held by the pool.
void pool_usage(int device, uint64_t* used, uint64_t* reserved);

// Stream-ordered allocation from the library's pool on the current device.  The pool never makes a call wait for
// a call on another stream, so under memory pressure the blocks such calls have freed can still
// be in flight: then the device is drained once and the allocation retried (not inside a stream
// capture, where the first error stands).
cudaError_t pool_malloc(void** p, size_t bytes, cudaStream_t s);
// Hands the memory the pool keeps cached between calls back to the device (after an ordinary
// allocation ran out of memory).
void trim_pool();

}  // namespace grgx
