// The server's planner (csrc/mbcg_plan.h) against building every cut: the same choice, and how many tiles it
// built for it.  argv: seed, compositions; or "cover": every fluid plane of long lattices in exactly one tile, at
// any depth.  Prints one line a composition: chosen index, exhaustive index, their
// predicted times, tiles built, tiles of the chosen cut, tiles of all cuts.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "mbcg_plan.h"

using namespace mbcg;

int cover() {
    double ns[BK_COUNT];
    for (double& v : ns) v = 1.0;
    for (int nz : {66000, 70003, 524282})
        for (int bcz : {MBCG_BC_PERIODIC, MBCG_BC_WALL})
            for (int z : {1, 5, 8, 12}) {
                const PlanLattice l{0, BK_Q27_F32, 6, 6, nz, bcz, 1 << 20};
                std::vector<TileItem> items;
                plan_tiles({l}, z, ns, 3.0, items);
                std::vector<char> seen(nz, 0);
                for (const TileItem& it : items) {
                    int zd0, zd1;
                    z_range(nz, bcz, plan_depth(l, z), it.t.bz, zd0, zd1);
                    for (int k = zd0; k < zd1; ++k) seen[k] += 1;
                }
                for (int k = 1; k < nz - 1; ++k)
                    if (seen[k] != 1) return std::printf("nz %d bcz %d z %d: plane %d in %d tiles\n", nz, bcz, z, k, seen[k]), 1;
            }
    return 0;
}

int main(int argc, char** argv) {
    if (argc > 1 && !std::strcmp(argv[1], "cover")) return cover();
    std::mt19937 rng(argc > 1 ? std::atoi(argv[1]) : 1);
    const int count = argc > 2 ? std::atoi(argv[2]) : 100;
    constexpr int n = sizeof(kCuts) / sizeof(kCuts[0]);
    auto uni = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(rng); };
    for (int c = 0; c < count; ++c) {
        std::vector<PlanLattice> L;
        double ns[BK_COUNT];
        for (double& v : ns) v = 1500.0 + 100.0 * uni(0, 20);
        // the first composition: as many 192^3 lattices as may be live
        const int live = c == 0 ? 64 : uni(1, 8);
        for (int i = 0; i < live; ++i) {
            const int e = uni(3, 7);
            const int size = 1 << e;
            PlanLattice l{i, uni(0, BK_COUNT - 1), 2 + size + uni(0, size), 2 + size + uni(0, size), 2 + size + uni(0, 3 * size),
                          uni(0, 2), 1 << 20};
            if (c == 0) l = {i, BK_Q27_F32_P, 194, 194, 194, 0, 1 << 20};
            L.push_back(l);
        }
        const double ovh = 0.5 * uni(2, 10);
        std::vector<TileItem> tiles, items;
        long long built = 0, all = 0;
        const Cut cut = plan_cut(L, ns, ovh, 152, tiles, &built);
        int chosen = 0, best = 0;
        double bt = 1e300, ct = 0.0;
        size_t ntiles = 0;
        for (int i = 0; i < n; ++i) {
            plan_tiles(L, kCuts[i].depth(), ns, ovh, items);
            all += static_cast<long long>(items.size());
            const double t = predict_ns(items, 152);
            if (t < plan_bound(L, kCuts[i].depth(), ns, ovh, 152) * (1 - 1e-9)) return std::printf("bound above the time\n"), 1;
            if (t < bt * 0.999) {
                bt = t;
                best = i;
            }
            if (kCuts[i].z == cut.z && kCuts[i].split == cut.split) {
                chosen = i;
                ct = t;
                ntiles = items.size();
                bool same = items.size() == tiles.size();
                for (size_t k = 0; same && k < items.size(); ++k)
                    same = items[k].t.slot == tiles[k].t.slot && items[k].t.bx == tiles[k].t.bx &&
                           items[k].t.by == tiles[k].t.by && items[k].t.bz == tiles[k].t.bz;
                if (!same) return std::printf("tiles are not those of the cut\n"), 1;
            }
        }
        std::printf("%d %d %.6f %.6f %lld %zu %lld\n", chosen, best, ct, bt, built, ntiles, all);
    }
    return 0;
}
