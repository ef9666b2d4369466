// The server's planner (csrc/mbcg_plan.h) against building every cut: the same choice, and how many tiles it
// built for it.  argv: seed, compositions.  Prints one line a composition: chosen index, exhaustive index, their
// predicted times, tiles built, tiles of the chosen cut, tiles of all cuts.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "mbcg_plan.h"

using namespace mbcg;

int main(int argc, char** argv) {
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
