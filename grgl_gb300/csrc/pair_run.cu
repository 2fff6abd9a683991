// Host side of the pair form: how a call's products are cut into tables and items, and the launches.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_plan.h"

namespace grgx {

namespace {

// Pattern rows held at a time: a table is written and gathered from before the next one.
constexpr size_t kPairTableBytes = 1ULL << 30;
// A share of the blocks (item) covers at most this much of a table.  The warps of a launch take
// the items of one share before those of the next, so about this much is gathered from at a time
// and mostly stays in L2 (N=200,000, M=250,000, K=64, at 96 MB / 48 / 192 / unshared, ms: float32, a 650 MB table, 3.63 /
// 3.84 / 3.78 / 3.86; int32 3.16 / 3.23 / 3.46 / 3.56; float64 8.06 / 8.27 / 7.90 / 8.44, K=32 4.01 / 4.12 / 4.14 / 4.29).
constexpr long long kPairItemBytes = 96LL << 20;
// Items per resident warp that even out the launch's end, and the fewest groups of four blocks
// that make an item worth its sum's trip through memory.
constexpr long long kPairItemsPerWarp = 8;
constexpr int kPairMinGroups = 16;
// UP: bytes of the height-0 rows' columns that a launch gathers from at a time (100 MB: float32 K=128 on
// 200,000 rows 3.95 ms against 3.63, 50 to 72 MB the same).
constexpr long long kPairSourceBytes = 64LL << 20;
// Blocks from which float64 sums eight pattern rows between folds, not four (error and time: pair_down_f64s.cu).
constexpr long long kPairLongRuns = 50;
// Most of a call's scratch unless a scope says less.
constexpr uint64_t kPairScratch = 6ULL << 30;

thread_local uint64_t t_limit = kPairScratch;

// Lanes per row.  A gather instruction costs the L1 about the same whichever of its lanes do nothing, so
// what counts is the instructions per row: its column tiles over the rows a warp's 32 lanes hold.  Ten
// lanes hold three rows where sixteen hold two, six hold five, five hold six; they are taken where they
// need at most 0.7 of the instructions of the layout's power of two, 0.8 where the additions of the
// idle lanes weigh too (compensated kinds; float32 DOWN only in a single tile).  Milliseconds on
// N=200,000, M=250,000, power of two against these:
//   float64 K=20 (10 vectors) UP 5.09 / 3.20  DOWN 4.00 / 3.01    K=36 (18) UP 10.1 / 6.2  DOWN 7.6 / 5.7
//   float64 K=24 (12)         UP 5.12 / 4.25  DOWN 4.07 / 3.89    float32 K=40 (10) UP 4.30 / 3.05  DOWN 3.55 / 2.85
//   int32 K=72 (18)           UP 7.20 / 6.01  DOWN 5.81 / 5.31    K=80 (20) UP 7.32 / 6.08  DOWN 5.78 / 5.41
// and past the line int32 K=20 (5) UP 1.86 / 2.10, K=48 (12) UP 3.74 / 4.12, float32 K=48 DOWN 3.58 / 3.85.
int pair_lanes(const Layout& L, bool up) {
    const long long vecs = L.stride / L.vw;
    auto cost = [&](int g) { return static_cast<double>((vecs + g - 1) / g) / (32 / g); };
    int best = L.g;
    for (int g : {10, 6, 5}) {
        if (L.vw * L.ssize != 16 || (g == 5 && up)) continue;
        const bool one = vecs <= g;
        const bool both = L.kind == Kind::F64S || (L.kind == Kind::F32C && (up || one));
        if (cost(g) <= (both ? 0.801 : 0.701) * cost(L.g) && cost(g) < cost(best)) best = g;
    }
    return best;
}

// Lanes per row for UP's gathers from the height-0 rows: as many as leave the columns of one tile
// in L2 (float64 K=64 on 200,000 rows: 102 MB at once, 60% L2 hits and 13.4 ms; in two tiles 11.3;
// float32 K=32 on 1,000,000: tiles of 32 MB 4.1, of 64 MB 2.7).
int source_lanes(const Layout& L, long long h0) {
    int g = pair_lanes(L, true);
    if (h0 * g * 16 > kPairSourceBytes) {
        g = L.g;
        while (g > 1 && h0 * g * 16 > kPairSourceBytes) g /= 2;
    }
    return g;
}

// Tiles that are not whole 128-byte lines bring their neighbours' parts of the lines into L2: the rows'
// columns are laid out tile by tile first where they don't all fit there.  UP on 1,000,000 samples and 50,000
// mutations in ms, from the rows as they are in 56 MB tiles, laid out in 64 MB tiles, and the split form:
// float32 K=32 9.2, 2.7 and 6.4, K=128 40.6, 10.4 and 18.0; float64 K=32 18.9, 6.3 and 11.3.  400,000 and
// 100,000: float32 K=96 8.2, 6.2 and 13.0; 200,000 and 100,000: 3.5, 3.4 and 6.7.
bool tile_sources(const Layout& L, long long h0) {
    const long long rowBytes = L.stride * L.ssize, tileBytes = source_lanes(L, h0) * 16LL;
    return L.vw * L.ssize == 16 && tileBytes < rowBytes && h0 * rowBytes > kPairSourceBytes &&
           (tileBytes % 128 != 0 || rowBytes % 128 != 0);
}

// dst[tile][row][lanes] from src[row][vecs], vectors of 16 bytes.  One pass over the rows: DRAM-bound.
__global__ void pair_source_kernel(const uint4* __restrict__ src, long long rows, int vecs, int lanes, uint4* __restrict__ dst) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows * vecs; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / vecs;
        const int v = static_cast<int>(i - r * vecs), tile = v / lanes;
        dst[(tile * rows + r) * lanes + v - tile * lanes] = src[i];
    }
}

// How compensated float32 adds DOWN pattern rows.  The sweep pre-sums four edges only in batches of
// edges without a row start, so the shorter the rows (two edges per block) and the fewer the columns, the
// fewer plain additions its sums pass.  Norm of the error against float64, 1e-8 of the norm, sweep / rounded
// pattern rows by FastTwoSum / by TwoSum / rows with their error; N(0,1) inputs, then standardized products:
//   200,000 samples and 3,000 variants (15 blocks), K=48 5.9 / - / - / 4.9 and 6.38 / - / - / 5.77, K=64 5.9 / - /
//     5.6 / - and 6.39 / - / 6.42 / -
//   200,000 and 10,000 (50),     K=18 6.0 / 5.7 / 5.6 / - and 7.17 / 7.35 / 7.12 / -
//   100,000 and 20,000 (100),    K=12 6.5 / 6.1 / 6.0 / - and 7.36 / 7.45 / 7.28 / -, K=100 6.8 / 5.9 / - / - and 8.2 / 7.5
//   200,000 and 250,000 (1,250), K=6 6.5 / - / 6.0 / - and 8.2 / - / 7.5 / -, K=12 6.4 / 5.8 / 5.9 / - and 8.2 / 7.6 / - / -
// Microseconds: 100,000 and 20,000 K=8 240 / - / 90 / 105, K=64 662 / 231 / 274 / -; 200,000 and 250,000 K=8 2260 / - /
// 858 / -, K=16 2757 / 1147 / 1329 / -.  The fastest kind that stays at or below the sweep's error in both is
// taken.  (Two rows pre-summed before a TwoSum take as long as two FastTwoSums and leave 6.4 where those leave 5.8.)
enum class DownSums { kOrdered, kSingle, kExact };
DownSums down_sums(const Layout& L, const PairPlan& P) {
    if (L.kind != Kind::F32C || L.vw == 1) return DownSums::kOrdered;
    const long long work = P.nblk * L.stride;
    if (work <= (P.nblk <= 50 ? 1000 : 800)) return DownSums::kExact;
    return work < 10000 || L.stride <= 8 ? DownSums::kSingle : DownSums::kOrdered;
}

// The layout that the DOWN pair kernels run with: pattern rows with their error take two columns a lane.
Layout down_layout(Layout L, const PairPlan& P) {
    if (down_sums(L, P) != DownSums::kExact) return L;
    L.vw = 2;
    const long long vecs = L.stride / 2;
    L.g = 1;
    while (L.g < 32 && L.g < vecs) L.g *= 2;
    return L;
}

template <typename F> void by_kind(const Layout& L, DownSums sums, F&& f) {
    switch (L.kind) {
    case Kind::U32: f(PairDownParams<uint32_t>{}, pair_down_u32); break;
    case Kind::XOR: f(PairDownParams<uint32_t>{}, pair_down_xor); break;
    case Kind::U64: f(PairDownParams<unsigned long long>{}, pair_down_u64); break;
    case Kind::F64: f(PairDownParams<double>{}, pair_down_f64); break;
    case Kind::F32C: f(PairDownParams<float>{}, sums == DownSums::kExact ? pair_down_f32cx
                                                    : sums == DownSums::kSingle ? pair_down_f32c1 : pair_down_f32c); break;
    case Kind::F32: f(PairDownParams<float>{}, pair_down_f32); break;
    case Kind::F64S: f(PairDownParams<DF>{}, pair_down_f64s); break;
    }
}

}  // namespace

PairScratchScope::PairScratchScope(uint64_t bytes) : saved_(t_limit) { t_limit = std::min(bytes, kPairScratch); }
PairScratchScope::~PairScratchScope() { t_limit = saved_; }
void set_pair_scratch(uint64_t bytes) { t_limit = bytes ? std::min(bytes, kPairScratch) : kPairScratch; }
size_t pair_scratch_limit() { return static_cast<size_t>(t_limit); }

PairDownRun pair_down_run(const Layout& call, const DevicePlan* dp, size_t limit) {
    const PairPlan& P = dp->pair;
    const Layout L = down_layout(call, P);
    const DownSums sums = down_sums(call, P);
    PairDownRun run;
    const int lanes = pair_lanes(L, false);
    run.tiles = static_cast<int>((L.stride / L.vw + lanes - 1) / lanes);
    PairDownCall shape;
    by_kind(L, sums, [&](auto p, auto fn) { fn(p, shape, L.vw, pair_lanes(L, false), sm_count(), nullptr); });
    const size_t rowBytes = static_cast<size_t>(L.stride) * shape.table_bytes;
    const size_t slotBytes = static_cast<size_t>(P.h0) * L.stride * shape.part_bytes;
    const size_t tableMost = std::min(kPairTableBytes, limit / 3);
    // sums held at a time: what the rest of the limit holds, one of them carried between ranges
    const long long slotsMost = static_cast<long long>((limit - tableMost) / slotBytes);
    const long long tiles = (P.h0 + shape.rows_per_warp - 1) / shape.rows_per_warp;
    const int groups = static_cast<int>((P.nblk + 3) / 4);
    auto patterns = [&](int g) { return P.pat_base[std::min<long long>(4LL * g, P.nblk)]; };
    for (int g0 = 0; g0 < groups;) {
        int g1 = g0 + 1;
        while (g1 < groups && static_cast<size_t>(patterns(g1 + 1) - patterns(g0)) * rowBytes <= tableMost) g1++;
        PairDownRun::Range r{};
        r.g0 = g0;
        r.g1 = g1;
        r.pat0 = patterns(g0);
        r.count = patterns(g1) - r.pat0;
        const long long carried = g0 > 0 ? 1 : 0;
        // (the columns of a tile are gathered together, so a share spans rowBytes / tiles per row)
        const long long share = static_cast<long long>(r.count * rowBytes / run.tiles) / kPairItemBytes + 1;
        const long long even = (kPairItemsPerWarp * shape.resident_warps + tiles - 1) / tiles;
        const long long most = std::min<long long>((g1 - g0) / kPairMinGroups, slotsMost - carried);
        const long long items = std::max(1LL, std::min(std::max(share, even), most));
        r.groups_per_item = static_cast<int>((g1 - g0 + items - 1) / items);
        r.items = (g1 - g0 + r.groups_per_item - 1) / r.groups_per_item;
        run.slots = std::max(run.slots, r.items + static_cast<int>(carried));
        run.table_bytes = std::max(run.table_bytes, static_cast<size_t>(r.count) * rowBytes);
        run.ranges.push_back(r);
        g0 = g1;
    }
    if (run.slots == 1) run.slots = 0;
    run.part_bytes = static_cast<size_t>(run.slots) * slotBytes;
    if (run.table_bytes + run.part_bytes > limit) run.ranges.clear();
    return run;
}

int launch_pair_down(const Layout& call, const DevicePlan* dp, const PairDownRun& run, void* vals, void* table, void* parts,
                     unsigned* work, cudaStream_t s, const int* gate) {
    const PairPlan& P = dp->pair;
    const Layout L = down_layout(call, P);
    int launches = 0;
    by_kind(L, down_sums(call, P), [&](auto p, auto fn) {
        PairDownCall c;
        fn(p, c, L.vw, pair_lanes(L, false), sm_count(), s);
        p.ids = reinterpret_cast<const uint2*>(P.ids);
        p.base = reinterpret_cast<const uint4*>(P.base);
        p.table = table;
        p.vals = static_cast<decltype(p.vals)>(vals);
        p.parts = run.slots ? parts : nullptr;
        p.rows = P.h0;
        p.stride = L.stride;
        p.groups = (P.nblk + 3) / 4;
        p.tiles = static_cast<unsigned>((P.h0 + c.rows_per_warp - 1) / c.rows_per_warp);
        p.gate = gate;
        p.long_runs = P.nblk >= kPairLongRuns;
        for (size_t i = 0; i < run.ranges.size(); i++) {
            const PairDownRun::Range& r = run.ranges[i];
            c.step = PairDownCall::kTable;
            c.nodes = P.pat_nodes + r.pat0;
            c.count = r.count;
            fn(p, c, L.vw, pair_lanes(L, false), sm_count(), s);
            c.step = PairDownCall::kGather;
            p.base0 = static_cast<unsigned>(r.pat0);
            p.group_begin = r.g0;
            p.group_end = r.g1;
            p.items = static_cast<unsigned>(r.items);
            p.groups_per_item = r.groups_per_item;
            p.part_begin = i > 0 ? 1 : 0;
            p.work = work + i * run.tiles;
            fn(p, c, L.vw, pair_lanes(L, false), sm_count(), s);
            launches += 2;
            if (run.slots == 0) continue;
            c.step = PairDownCall::kFinish;
            c.parts = r.items + p.part_begin;
            c.onto = i + 1 == run.ranges.size();
            if (c.onto || c.parts > 1) {
                fn(p, c, L.vw, pair_lanes(L, false), sm_count(), s);
                launches++;
            }
        }
    });
    return launches;
}

PairUpRun pair_up_run(const Layout& L, const DevicePlan* dp, size_t limit) {
    const std::vector<PairPlan::Segment>& seg = dp->pair.segments;
    PairUpRun run;
    const size_t rowBytes = static_cast<size_t>(L.stride) * L.ssize, most = std::min(kPairTableBytes, limit);
    for (size_t s0 = 0; s0 + 1 < seg.size();) {
        size_t s1 = s0 + 1;
        while (s1 + 1 < seg.size() && static_cast<size_t>(seg[s1 + 1].row0 - seg[s0].row0) * rowBytes <= most) s1++;
        run.ranges.push_back({s0, s1});
        run.table_bytes = std::max(run.table_bytes, static_cast<size_t>(seg[s1].row0 - seg[s0].row0) * rowBytes);
        s0 = s1;
    }
    if (run.table_bytes > limit) run.ranges.clear();
    if (tile_sources(L, dp->pair.h0)) {
        const long long g = source_lanes(L, dp->pair.h0), tiles = (L.stride / L.vw + g - 1) / g;
        const size_t bytes = static_cast<size_t>(tiles * g * dp->pair.h0) * 16;
        if (run.table_bytes + bytes <= limit) run.source_bytes = bytes;
    }
    return run;
}

PairRuns pair_runs(grgx_graph* g, DevicePlan* dp, const Layout& L, bool down, cudaStream_t s) {
    PairRuns r;
    if (!use_pair_form(g, dp, L, down, s)) return r;
    const size_t limit = pair_scratch_limit();
    if (down) {
        r.down = pair_down_run(L, dp, limit);
        return r;
    }
    if (L.kind == Kind::F32C) r.up_state_bytes = static_cast<size_t>(g->host->num_nodes - dp->pair.h0) * L.stride * L.asize;
    if (r.up_state_bytes < limit) r.up = pair_up_run(L, dp, limit - r.up_state_bytes);
    return r;
}

int launch_pair_up(const Layout& L, const DevicePlan* dp, const PairUpRun& run, void* vals, void* table, void* state,
                   int rmw, cudaStream_t s, const int* gate) {
    const PairPlan& P = dp->pair;
    int launches = 0;
    const int all = pair_lanes(L, true), g = source_lanes(L, P.h0);
    char* const tiled = run.source_bytes ? static_cast<char*>(table) + run.table_bytes : nullptr;
    if (tiled) {
        pair_source_kernel<<<sm_count() * 8, 256, 0, s>>>(static_cast<const uint4*>(vals), P.h0,
                                                          static_cast<int>(L.stride / L.vw), g, reinterpret_cast<uint4*>(tiled));
        launches++;
    }
    const size_t rowBytes = static_cast<size_t>(L.stride) * L.ssize;
    bool few = P.nfew > 0;  // (with the first range)
    for (const PairUpRun::Range& r : run.ranges) {
        const PairPlan::Segment &a = P.segments[r.s0], &b = P.segments[r.s1];
        // table rows count from the first segment's first one, the nodes' from height 1 on
        char* t = static_cast<char*>(table) - static_cast<size_t>(a.row0) * rowBytes;
        char* nodes = static_cast<char*>(vals) + static_cast<size_t>(P.h0) * rowBytes;
        auto lists = [&](const PairList* list, long long count, const uint32_t* adj, bool second, bool rows) {
            if (count == 0) return;
            auto go = [&](auto p, auto fn) {
                p.lists = list;
                p.count = count;
                p.adj = adj;
                p.src = reinterpret_cast<decltype(p.src)>(!rows ? t : tiled ? tiled : static_cast<char*>(vals));
                const int lanes = rows ? g : all;
                p.src_stride = rows && tiled ? static_cast<long long>(g) * L.vw : L.stride;
                p.tile_step = (rows && tiled ? P.h0 : 1) * lanes * L.vw;
                p.table = reinterpret_cast<decltype(p.table)>(t);
                p.dst = reinterpret_cast<decltype(p.dst)>(nodes);
                p.rmw = rmw;
                p.state = state;
                p.second = second ? 1 : 0;
                p.stride = L.stride;
                p.gate = gate;
                fn(p, L.vw, lanes, s);
            };
            switch (L.kind) {
            case Kind::U32: go(PairUpParams<uint32_t>{}, pair_up_u32); break;
            case Kind::XOR: go(PairUpParams<uint32_t>{}, pair_up_xor); break;
            case Kind::U64: go(PairUpParams<unsigned long long>{}, pair_up_u64); break;
            case Kind::F64: go(PairUpParams<double>{}, pair_up_f64); break;
            case Kind::F32C: go(PairUpParams<float>{}, pair_up_f32c); break;
            case Kind::F32: go(PairUpParams<float>{}, pair_up_f32); break;
            case Kind::F64S: go(PairUpParams<DF>{}, pair_up_f64s); break;
            }
            launches++;
        };
        lists(P.pat_lists + a.pat0, b.pat0 - a.pat0, P.pat_adj, false, true);
        if (few) lists(P.few_lists, P.nfew, P.few_adj, true, true);
        few = false;
        lists(P.node_lists + a.node0, b.node0 - a.node0, P.node_adj, true, false);
        lists(P.top_lists + a.top0, b.top0 - a.top0, P.top_adj, true, false);
    }
    return launches;
}

}  // namespace grgx
