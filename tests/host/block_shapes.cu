// Which tiles runs are cut into (heat_block.cuh, heatvar_block.cuh).  Reads lines
// "list nx ny levels" and answers with the shapes C,R,nw (stream: 0,0,0) of the
// launches of such a run on 148 SMs; "list 0 0 0": with all the shapes of the list.
// Built and run by tests/test_host_block_shapes.py (nvcc, no GPU needed).
#include <cstdio>
#include <cstring>

#include "../../pysweep_b200/csrc/heatvar_block.cuh"

using namespace psb;

constexpr int kSms = 148;

static void show(const TileShape& t) { printf("%d,%d,%d ", t.C, t.R, t.nw); }

template <int N, class Plan, class Best>
static void launches(const TileShape (&shapes)[N], int levels, int step, bool streams, Plan&& plan,
                     Best&& best)
{
    if (!levels) {
        for (const TileShape& t : shapes) show(t);
        if (streams) show(TileShape{0, 0, 0, 0});
        return;
    }
    const BlockPlan p = plan();
    for (int left = levels; left > 0;) {
        const int T = plan_next(p, left, step);
        show(p.stream && T == kStreamT ? TileShape{0, 0, 0, 0} : best(T));
        left -= T;
    }
}

template <int N>
static void heat(const TileShape (&shapes)[N], const BlockGrids& g, int levels, int step,
                 const TileCost& plan_cost, const TileCost& cost)
{
    double us;
    launches(shapes, levels, step, true,
             [&] { return plan_block(shapes, g, levels, step, kTileMaxT, kSms, plan_cost); },
             [&](int T) { return best_tile(shapes, T, g, kSms, &us, cost); });
}

template <int ROLE, int N>
static void var(const TileShape (&shapes)[N], const BlockGrids& g, int levels)
{
    double us;
    launches(shapes, levels, 1, false, [&] { return plan_var<ROLE>(g, levels, kSms); },
             [&](int T) { return best_tile(shapes, T, g, kSms, &us, var_cost<ROLE>()); });
}

int main()
{
    char list[16];
    int nx, ny, n;
    while (scanf("%15s %d %d %d", list, &nx, &ny, &n) == 4) {
        const BlockGrid one{nx, ny};
        const BlockGrids g{&one, 1};
        double us;
        auto is = [&](const char* s) { return !strcmp(list, s); };
        if (is("fe")) heat(kTilesFE, g, n, 1, TileCost{}, TileCost{});
        else if (is("f32")) heat(kTilesFE, g, n, 1, kCostF32, TileCost{});
        else if (is("rk2")) heat(kTilesRK2, g, n, 2, kCostRK2, kCostRK2);
        else if (is("forward")) var<VAR_FORWARD>(kTilesVar, g, n);
        else if (is("recompute")) var<VAR_RECOMPUTE>(kTilesVar, g, n);
        else if (is("adjoint")) var<VAR_MU>(kTilesAdj, g, n);
        else if (is("backward"))
            launches(kTilesBack, n, 1, false, [&] { return plan_back(g, n, kSms); },
                     [&](int T) { return best_back(T, g, kSms, &us); });
        else return 1;
        printf("\n");
    }
    return 0;
}
