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

namespace grgx {

// Graphs with fewer edges between height-0 nodes and parents keep the other forms.
constexpr long long kPairMinEdges = 1LL << 22;
// The form is used when its gathers -- one per block and height-0 node, kPairPatternCost per
// pattern (two reads, a write and the table's own traffic) -- are at most this share of one per edge.
constexpr double kPairPatternCost = 4.0;
constexpr double kPairMaxCost = 0.75;

struct PairPlan {
    bool tried = false;   // the analysis ran (once per graph)
    bool usable = false;  // ... and found the form worth using
    long long h0 = 0;     // height-0 nodes (new ids 0 .. h0-1)
    long long nblk = 0;
    long long npat = 0;
    std::vector<long long> pat_base;  // first pattern of each block (nblk + 1)
    unsigned* base = nullptr;         // the same on the device, padded to whole groups of four blocks
    uint2* pat_nodes = nullptr;       // the pattern's two parents (new ids, INVALID_NODE = none)
    // DOWN: each height-0 node's pattern within each block (0: the empty pair), 16 bits, ordered
    // [tile of 32 nodes][group of four blocks][node][block]: a node's four ids are one 8-byte load
    unsigned short* ids = nullptr;
};

}  // namespace grgx
