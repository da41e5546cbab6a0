// How a contraction shares its (observer, source) pairs out: ob observers a
// block of `threads`, threads / ob slices of each source tile, the tiles dealt
// over the `ranks` blocks of a cluster.
#pragma once
#include "common.cuh"

namespace mbem {

struct ConSplit {
    int ob, ranks;
};

// The split whose fullest SM has the fewest FP64 warp instructions: a block
// pays `setup` of them per 32 sources for their records and `pair` per 32 pairs
// (the FP64 pipe is the bound: a warp instruction takes 16 cycles of an SM).
// Small observer counts want few observers a block and wide clusters (48
// observers x 6,912 sources: 6 blocks of whole source lists took 10 ms); large
// ones whole blocks of observers, whose records are made least often. Fewer than
// about five warps an SM leave the pipe waiting for results; beyond a few blocks
// an SM the scheduler evens them out.
inline ConSplit contract_split(int64_t nf, int64_t ns, int threads, int max_ob, int tile, double pair, double setup) {
    constexpr int sms = 152;
    static const int obs[] = {1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 48, 64};
    ConSplit best = {max_ob, 1};
    double cost = 1e300;
    for (int ranks = 1; ranks <= 8; ranks *= 2) {
        if (ranks > 1 && (int64_t)tile * (ranks / 2) >= ns) break;      // a rank would have no source
        for (int ob : obs) {
            if (ob > max_ob || (ob > 1 && ob / 2 >= nf)) continue;
            const int slices = threads / ob;
            const int64_t blocks = ceil_div(nf, ob) * ranks;
            const double tiles = (double)ceil_div(ceil_div(ns, tile), ranks);
            const double in_tile = (double)lmin(tile, ceil_div(ns, ranks));
            const double per = tiles * (setup * (tile / 32.0 > 1.0 ? tile / 32.0 : 1.0) +
                                        pair * (threads / 32) * (double)ceil_div((int64_t)in_tile, slices));
            double rounds = blocks > 6 * sms ? (double)blocks / sms + 0.5 : (double)ceil_div(blocks, sms);
            if (rounds * (threads / 32) < 5.0) rounds = 5.0 / (threads / 32);
            const double c = rounds * per;
            if (c < cost * 0.999) {
                cost = c;
                best.ob = ob;
                best.ranks = ranks;
            }
        }
    }
    return best;
}

}  // namespace mbem
