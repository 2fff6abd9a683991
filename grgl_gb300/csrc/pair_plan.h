// Pair form of the edges between height-0 nodes and their parents (internal).
//
// Runs.  Take the nodes that have height-0 children in original id order.  A run is a maximal
// stretch of them whose height-0 children are disjoint, so a height-0 node has at most one parent
// per run (in a window-tree graph a run is a window).  Two consecutive runs form a block: within
// it a height-0 node is known by its pair (parent in the first run or none, parent in the second
// or none), and with far more height-0 nodes than nodes per run most share their pair with many
// others.  Each distinct pair of a block is a pattern.
//   DOWN  pattern row = sum of its (at most two) parents' rows; a height-0 node adds one pattern
//         row per block instead of one row per edge
//   UP    pattern row = sum over the height-0 nodes that have the pair; a parent adds its
//         patterns' rows instead of one row per height-0 child
// Either way the row gathers of these edges -- what the traversals cost -- are halved, plus a few
// per pattern.
#pragma once
#include <cstdint>
#include <vector>

#include "launch.h"

namespace grgx {

// Graphs with fewer edges between height-0 nodes and parents keep the other forms: their calls are
// a chain of launches either way (N=20,000, M=5,000, 1e6 edges: int32 K=5 UP 77 us against 56 in
// pair form, DOWN 57 against 47; building it takes 4 ms).
constexpr long long kPairMinEdges = 1000000;
// The form is used when its gathers -- one per block and height-0 node, kPairPatternCost per
// pattern (two reads, a write and the table's own traffic) -- are at most this share of one per edge.
constexpr double kPairPatternCost = 4.0;
// (N=5,000, M=50,000: 0.86; float64 K=20 UP 0.32 against 0.20 ms, DOWN 0.172 against 0.160.)
constexpr double kPairMaxCost = 0.9;

// UP: lists (a pattern's height-0 nodes, a node's table rows) are summed in pieces of at most this
// many, each with a row of its own in the table; it bounds how long one group of lanes works on one.
constexpr long long kPairPiece = 256;
// UP: nodes with at most this many height-0 children sum them directly, with the nodes' own additions.  Over
// pattern rows, which compensated float32 rounds, such nodes ended up to 1.3e-7 of sum |terms| off, directly
// 6.0e-8 as in the sweep (N=200,000, M=250,000, K=8, N(0,1) inputs; float64 7.7e-15 and 3.7e-15).  They hold few
// of the edges: 1277 and 1261 us there, float32 K=40 3052 and 3065, N=20,000, M=50,000 203 and 208.
constexpr unsigned kPairFew = 32;
// UP: a list's destination row, or the complement of a table row, is an int.
constexpr long long kPairMostRows = 0x3fffffff;
// Blocks whose lists are sorted by length together, longest first (the order they are launched in).
constexpr long long kPairSegment = 64;

// One block: its runs' first positions in the sequence of nodes with height-0 children, and their
// node counts (n1 = 0: a block of one run).
struct PairBlock {
    int run, q0, q1, n0, n1;
};

struct PairPlan {
    bool refused = false;  // the analysis found the form not worth using (decided once per graph)
    bool usable = false;   // ... or worth it, and the arrays of some direction are built
    bool down_tried = false, up_tried = false;  // a build of the direction has succeeded or failed for good
    // Written once, before `usable` is set: calls read these after use_pair_form has let go of the graph's
    // lock, also while another thread's first call of the other direction builds that direction's arrays.
    long long h0 = 0;     // height-0 nodes (new ids 0 .. h0-1)
    long long nblk = 0;
    long long npat = 0;
    std::vector<long long> pat_base;  // first pattern of each block (nblk + 1)
    // kept for the second direction's arrays: the sequence (UP rows), its runs and blocks, and
    // each UP row's height-0 children
    std::vector<int> seq, run;
    std::vector<PairBlock> blocks;
    std::vector<unsigned> low;
    // DOWN, on the first DOWN call:
    bool down_built = false;
    unsigned* base = nullptr;         // pat_base on the device, padded to whole groups of four blocks
    uint2* pat_nodes = nullptr;       // the pattern's two parents (new ids, INVALID_NODE = none)
    // each height-0 node's pattern within each block (0: the empty pair), 16 bits, ordered
    // [tile of 32 nodes][group of four blocks][node][block]: a node's four ids are one 8-byte load
    unsigned short* ids = nullptr;
    // UP, on the first UP call: lists of height-0 nodes (the patterns' pieces, a table row each), of
    // table rows (the nodes, and the pieces of nodes with many), and of such pieces' rows (those
    // nodes), by segments of blocks.
    bool up_built = false;
    struct Segment {
        long long row0 = 0;                       // first table row
        long long pat0 = 0, node0 = 0, top0 = 0;  // first list of each kind
    };
    std::vector<Segment> segments;                // + the end
    PairList *pat_lists = nullptr, *node_lists = nullptr, *top_lists = nullptr;
    uint32_t *pat_adj = nullptr, *node_adj = nullptr, *top_adj = nullptr;
    // nodes of few height-0 children: lists of those, by length
    long long nfew = 0;
    PairList* few_lists = nullptr;
    uint32_t* few_adj = nullptr;
};

}  // namespace grgx
