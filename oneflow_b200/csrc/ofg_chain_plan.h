// The schedule of one chained LU-SGS sweep (ofg_chain.cuh), formed on the host:
// edge slots [level][j-th edge][cell of the level], and for each edge where the
// sweep finds its neighbour's increment, in the ring that the cluster's blocks
// keep in shared memory or, further back, in global memory.  Plain C++, so
// that the schedule's orders can be checked without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace ofg {

// warps of a level and groups of them in a block; ring positions
constexpr int kChainWarps = 6, kChainGroups = 2, kChainThreads = 32 * kChainWarps * kChainGroups;
// arrivals that a level's phase of a block's mbarrier waits for: one of every warp of its group (chain_run)
constexpr int kChainArrivals = kChainWarps;
constexpr int kChainRing = 4096, kChainMaxBlocks = 16;
constexpr int kChainLevel = 16384;      // most cells of a level: their bytes are counted on an mbarrier (chain_run)
constexpr int kChainNone = INT32_MIN;   // an empty edge slot

struct SweepPlan {
    std::vector<int> lev;    // per level {first position, cells, first slot, slots per cell}
    std::vector<int> ref;    // [slots] ring slot of the neighbour, ~neighbour when the ring does not hold it, kChainNone
    std::vector<int> edge;   // [slots] {face | side << 31, neighbour, cell, -}; -1 on an empty slot
    long long slots = 0;
    int far = 0;             // 1: some neighbour comes from global memory; 2: and soon after it is written
    bool fits = true;        // false: the sweep cannot run chained (nothing else is set then)
};

// order[nCells]: the cells level after level, off[levels + 1] the levels; nbOff /
// nbl: each cell's edges in ascending face id, {face | side << 31, neighbour}.
//
// The ring holds position p of the level order in slot p mod kChainRing.  Levels
// are ordered one after the other, the cells of a level are not.  So an edge of
// level l takes its neighbour from the ring where every other write to the slot
// is ordered against this read:
// - near: later positions up to the end of level l have other slots;
// - alone: so have the earlier positions of the neighbour's own level (in a level
//   wider than the ring their write may arrive last).
inline void plan_sweep(int nCells, const std::vector<int> &order, const std::vector<int> &off, const std::vector<int> &nbOff,
                       const std::vector<int> &nbl, SweepPlan &P) {
    const int nlev = int(off.size()) - 1;
    std::vector<int> pos(nCells), at(nCells);
    P.lev.assign(4 * (size_t)nlev, 0);
    for (int l = 0; l < nlev; ++l) {
        int deg = 0;
        for (int k = off[l]; k < off[l + 1]; ++k) {
            const int i = order[k];
            pos[i] = k; at[i] = l;
            deg = std::max(deg, nbOff[i + 1] - nbOff[i]);
        }
        int *m = &P.lev[4 * (size_t)l];
        m[0] = off[l]; m[1] = off[l + 1] - off[l]; m[2] = int(P.slots); m[3] = deg;
        P.slots += (long long)deg * m[1];
        P.fits = P.fits && P.slots <= INT32_MAX / 4 && m[1] <= kChainLevel;
        if (!P.fits) return;
    }
    P.ref.assign(P.slots, kChainNone);
    P.edge.assign(4 * P.slots, -1);
    for (int l = 0; l < nlev; ++l) {
        const int *m = &P.lev[4 * (size_t)l];
        for (int t = 0; t < m[1]; ++t) {
            const int i = order[m[0] + t];
            size_t s = (size_t)m[2] + t;
            for (int q = nbOff[i]; q < nbOff[i + 1]; ++q, s += m[1]) {   // ascending face id
                const int nb = nbl[2 * (size_t)q + 1];
                const bool near = pos[nb] + kChainRing >= off[l + 1], alone = pos[nb] - kChainRing < off[at[nb]];
                P.ref[s] = near && alone ? pos[nb] & (kChainRing - 1) : ~nb;
                // A global copy written after its signal, in level a, is
                // released by its warp's next arrival, in level a +
                // kChainGroups; the other blocks learn of that arrival by
                // the word its block sends in the level after, so their
                // cells may read the copy from the level after that on.
                if (P.ref[s] < 0) P.far = std::max(P.far, l <= at[nb] + kChainGroups + 1 ? 2 : 1);
                int *e = &P.edge[4 * s];
                e[0] = nbl[2 * (size_t)q]; e[1] = nb; e[2] = i;
            }
        }
    }
}

}  // namespace ofg
