// mbcg_plan.h -- the server's planner: how deep the tiles of a batch composition are cut along z.  Host code.
#pragma once

#include <algorithm>
#include <functional>
#include <vector>

#include "mbcg_batch.h"

namespace mbcg {

struct PlanLattice {
    int slot, kind;
    int nx, ny, nz, bcz;
    int max_depth; // max_zchunk
};

struct TileItem {
    BatchTile t;
    int kind;
    double cost; // predicted ns
};

// Tiles z planes deep (8 or more), or such tiles in `split` parts, which compositions too small to fill the
// SMs take (8 requests of 16 to 48 nodes across: 4.6 ms, 5.5 without the parts).
struct Cut {
    int z, split;
    int depth() const { return (z + split - 1) / split; }
};
constexpr Cut kCuts[] = {{8, 8}, {8, 4}, {8, 3}, {8, 2}, {12, 2}, {8, 1}, {12, 1}, {16, 1}, {24, 1},
                         {32, 1}, {48, 1}, {64, 1}, {96, 1}, {128, 1}, {192, 1}, {256, 1}, {512, 1}};

inline int plan_bcz(const PlanLattice& l) { return batch_bcz(l.kind, l.bcz); }
// Depth of a lattice's tiles for a target z: equal chunks of at most z planes, or more where the chunks and two
// end tiles would outgrow a tile's 16-bit index.
inline int plan_depth(const PlanLattice& l, int z) {
    const int nzf = l.nz - 2 - 2 * z_cap(l.nz, plan_bcz(l));
    constexpr int kMaxChunks = 0xffff - 2;
    const int zmax = std::max(std::min(z, l.max_depth), (nzf + kMaxChunks - 1) / kMaxChunks);
    const int nch = std::max(1, (nzf + zmax - 1) / zmax);
    return (nzf + nch - 1) / nch;
}
inline int plan_gx(const PlanLattice& l) { return (l.nx - 2 + kStepTileX - 1) / kStepTileX; }
inline int plan_gy(const PlanLattice& l) {
    const int rows = batch_rows(l.kind) - 2;
    return (l.ny - 2 + rows - 1) / rows;
}

// Tiles of every lattice for a target depth z, longest first.  A tile costs (planes + 2 warm-up planes +
// overhead) x the calibrated time of one plane of its body.
inline void plan_tiles(const std::vector<PlanLattice>& lattices, int z, const double* plane_ns, double ovh,
                       std::vector<TileItem>& items) {
    items.clear();
    for (const PlanLattice& l : lattices) {
        const int gx = plan_gx(l), gy = plan_gy(l), bcz = plan_bcz(l), depth = plan_depth(l, z);
        const int gz = z_tiles(l.nz, bcz, depth);
        for (int bz = 0; bz < gz; ++bz) {
            int zd0, zd1;
            z_range(l.nz, bcz, depth, bz, zd0, zd1);
            const double planes = zd1 - zd0 + 2 + ovh;
            for (int by = 0; by < gy; ++by)
                for (int bx = 0; bx < gx; ++bx)
                    items.push_back({BatchTile{static_cast<uint16_t>(l.slot), static_cast<uint16_t>(bx),
                                               static_cast<uint16_t>(by), static_cast<uint16_t>(bz)},
                                     l.kind, planes * plane_ns[l.kind]});
        }
    }
    // longest tiles first: the atomic queues then run a greedy longest-processing-time schedule
    std::stable_sort(items.begin(), items.end(), [](const TileItem& a, const TileItem& b) {
        if (a.cost != b.cost) return a.cost > b.cost;
        return a.kind < b.kind;
    });
}

// Predicted duration of one launch: the greedy schedule of the sorted tiles on nsm CTAs.
inline double predict_ns(const std::vector<TileItem>& items, int nsm) {
    std::vector<double> load(std::max(1, nsm), 0.0);
    std::make_heap(load.begin(), load.end(), std::greater<double>());
    for (const TileItem& it : items) {
        std::pop_heap(load.begin(), load.end(), std::greater<double>());
        load.back() += it.cost;
        std::push_heap(load.begin(), load.end(), std::greater<double>());
    }
    return *std::max_element(load.begin(), load.end());
}

// What predict_ns() returns at least for a target depth z: all the work spread evenly, or the longest tile.
inline double plan_bound(const std::vector<PlanLattice>& lattices, int z, const double* plane_ns, double ovh, int nsm) {
    double work = 0.0, longest = 0.0;
    for (const PlanLattice& l : lattices) {
        const int bcz = plan_bcz(l), depth = plan_depth(l, z);
        const double tiles = z_tiles(l.nz, bcz, depth);
        work += static_cast<double>(plan_gx(l)) * plan_gy(l) * (l.nz - 2 + tiles * (2 + ovh)) * plane_ns[l.kind];
        longest = std::max(longest, (depth + 2 + ovh) * plane_ns[l.kind]);
    }
    return std::max(work / std::max(1, nsm), longest);
}

// The cut with the shortest predicted launch (of cuts within 0.1 %, the earlier in kCuts), and its tiles.  Tiles
// are built, sorted and scheduled only for cuts that can still be the best: first the one with the least bound,
// then those whose bound is not above its time.  64 lattices of 192^3 have 774 thousand tiles one plane deep:
// building every cut's takes 48 ms of a Grace core with the server's lock held, this 0.2 ms (8 small lattices: 0.06
// and 0.01 ms).  built: how many tiles that made.
inline Cut plan_cut(const std::vector<PlanLattice>& lattices, const double* plane_ns, double ovh, int nsm,
                    std::vector<TileItem>& tiles, long long* built = nullptr) {
    constexpr int n = sizeof(kCuts) / sizeof(kCuts[0]);
    double bound[n];
    int first = 0;
    for (int i = 0; i < n; ++i) {
        bound[i] = plan_bound(lattices, kCuts[i].depth(), plane_ns, ovh, nsm);
        if (bound[i] < bound[first]) first = i;
    }
    std::vector<TileItem> items;
    long long made = 0;
    plan_tiles(lattices, kCuts[first].depth(), plane_ns, ovh, tiles);
    made += static_cast<long long>(tiles.size());
    const double limit = predict_ns(tiles, nsm);
    double best = 1e300;
    int at = first;
    for (int i = 0; i < n; ++i) {
        if (i != first && bound[i] * 0.999 > limit) continue;
        double t = limit;
        if (i != first) {
            plan_tiles(lattices, kCuts[i].depth(), plane_ns, ovh, items);
            made += static_cast<long long>(items.size());
            t = predict_ns(items, nsm);
        }
        if (t < best * 0.999) {
            best = t;
            at = i;
        }
    }
    if (at != first) plan_tiles(lattices, kCuts[at].depth(), plane_ns, ovh, tiles);
    if (built) *built = made;
    return kCuts[at];
}

} // namespace mbcg
