// Cuts the tiles of a plan's graphs into the CTA shares of the sweep's first phase
// (host code without CUDA, so that it can be checked without a GPU).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

namespace egpr {

constexpr int kCutTileEntries = 256;  // entries of a tile

// A CTA's piece of phase 1: tiles [tile0, tile1) of one block of one graph.
struct GatherUnit {
    int32_t graph;
    int32_t block;
    int32_t tile0, tile1;
};

struct CutGraph {
    const int32_t* block_tile;  // first tile of each block (nblocks + 1)
    const int32_t* block_pair;  // first pair of each block (nblocks + 1)
    int32_t nblocks;
    int32_t chunk_shift;        // log2 of the tiles per chunk
    int32_t pair_cost;          // of a pair, in entries
};

// Equal shares of the cost, contiguous in (graph, block, tile).  cta_unit: first unit of
// each CTA (grid + 1).  Units begin and end on chunk boundaries of their block (or at
// the block's end): the layout ends runs there, and a unit carries nothing over.
inline void cut_gather_units(const CutGraph* graphs, int32_t count, int32_t grid, std::vector<GatherUnit>& units,
                             std::vector<int32_t>& cta_unit) {
    double cost = 0.0;
    for (int32_t gi = 0; gi < count; ++gi) {
        const CutGraph& g = graphs[gi];
        cost += (double)g.block_tile[g.nblocks] * kCutTileEntries + (double)g.pair_cost * g.block_pair[g.nblocks];
    }
    units.clear();
    cta_unit.assign(1, 0);
    const double share = cost / grid;
    double used = 0.0;  // of the current CTA's share
    for (int32_t gi = 0; gi < count; ++gi) {
        const CutGraph& g = graphs[gi];
        for (int32_t b = 0; b < g.nblocks; ++b) {
            const int32_t t1 = g.block_tile[b + 1];
            int32_t t = g.block_tile[b];
            const double per_tile =
                kCutTileEntries + (double)g.pair_cost * (g.block_pair[b + 1] - g.block_pair[b]) / std::max(1, t1 - t);
            while (t < t1) {
                const bool last = (int32_t)cta_unit.size() >= grid;  // the last CTA takes the rest
                if (!last && used >= share) {
                    cta_unit.push_back((int32_t)units.size());
                    used = 0.0;
                    continue;
                }
                // whole chunks, one at least: what is left of the share may be less than the
                // thousandth of a tile that the rounding gives away
                const int64_t chunk = (int64_t)1 << g.chunk_shift;
                int64_t take = last ? t1 - t : (int64_t)((share - used) / per_tile + 0.999);
                take = std::max(chunk, (take + chunk - 1) & ~(chunk - 1));
                take = std::min<int64_t>(take, t1 - t);
                units.push_back(GatherUnit{gi, b, t, t + (int32_t)take});
                used += per_tile * (double)take;
                t += (int32_t)take;
            }
        }
    }
    while ((int32_t)cta_unit.size() <= grid) cta_unit.push_back((int32_t)units.size());
}

}  // namespace egpr
