// Host-side check of the plans beside plain heat's (heat_block.cuh,
// heatvar_block.cuh, euler_march.cuh): with every cost that is in use, each launch of
// a plan has a tile with exact rows and columns left, whole lanes of halo, no more
// warps than its kernel allows and shared memory that fits; Euler's strips cover the
// rows.  Built and run by tests/test_host_block_costs.py (nvcc, no GPU needed).
#include <cstdio>

#include "../../pysweep_b200/csrc/euler_march.cuh"
#include "../../pysweep_b200/csrc/heatvar_block.cuh"

using namespace psb;

static bool sound(const char* what, const TileShape& t, int T, int nx, int ny, double us, size_t smem,
                  int warps)
{
    const int halo = (32 * t.C - tile_vw(t, T)) / 2;
    if (tile_vh(t, T) >= 2 && tile_vw(t, T) >= 8 && halo >= T && halo % t.C == 0 && t.nw <= warps &&
        us > 0 && us < 1e300 && smem <= 227 * 1024)
        return true;
    printf("%s %dx%d T %d: %d columns, %d rows, %d warps, %zu bytes\n", what, nx, ny, T, t.C, t.R, t.nw, smem);
    return false;
}

// every launch of a run of n levels
template <class Best>
static bool run(const BlockPlan& p, int n, int step, int maxT, Best&& best)
{
    if (p.T < step || p.T % step || p.T > maxT || (p.stream && p.T != kStreamT)) {
        printf("plan of %d levels: T %d\n", n, p.T);
        return false;
    }
    for (int left = n; left > 0;) {
        const int T = plan_next(p, left, step);
        if (T < 1 || T > left || T > maxT) {
            printf("launch of %d of %d levels\n", T, left);
            return false;
        }
        if (!(p.stream && T == kStreamT) && !best(T)) return false;
        left -= T;
    }
    return true;
}

template <int ROLE, int N>
static bool var(const char* what, const TileShape (&shapes)[N], const BlockGrid& g, int n, int sms)
{
    const BlockGrids gs{&g, 1};
    return run(plan_var<ROLE>(gs, n, sms), n, 1, kTileMaxT, [&](int T) {
        double us;
        const TileShape t = best_tile(shapes, T, gs, sms, &us, var_cost<ROLE>());
        return sound(what, t, T, g.nx, g.ny, us, tile_smem<2>(t.nw), t.maxw);
    });
}

int main()
{
    for (int sms : {1, 16, 132, 148})
        for (int nx : {3, 4, 8, 24, 50, 112, 160, 250, 481, 1120, 2048, 5000, 8192, 30000})
            for (int ny : {4, 8, 30, 64, 112, 160, 390, 1000, 2048, 8192, 20000}) {
                const BlockGrid g{nx, ny};
                const BlockGrids gs{&g, 1};
                double us;
                for (int n : {1, 2, 3, 7, 8, 9, 15, 16, 17, 64, 100, 5000}) {
                    const bool f32 = run(plan_block(kTilesFE, gs, n, 1, kTileMaxT, sms, kCostF32), n, 1, kTileMaxT,
                                         [&](int T) {
                                             const TileShape t = best_tile(kTilesFE, T, gs, sms, &us);
                                             return sound("float32", t, T, nx, ny, us, tile_smem<4>(t.nw), t.maxw);
                                         });
                    const int even = n - n % 2;
                    const bool rk2 =
                        !even || run(plan_block(kTilesRK2, gs, even, 2, kTileMaxT, sms, kCostRK2), even, 2, kTileMaxT,
                                     [&](int T) {
                                         const TileShape t = best_tile(kTilesRK2, T, gs, sms, &us, kCostRK2);
                                         return sound("two stages", t, T, nx, ny, us, tile_smem<4>(t.nw), t.maxw);
                                     });
                    const bool back = run(plan_back(gs, n, sms), n, 1, kBackMaxT, [&](int T) {
                        const TileShape t = best_back(T, gs, sms, &us);
                        return sound("backward", t, T, nx, ny, us, back_smem(t.R, t.nw, T), t.maxw);
                    });
                    if (!f32 || !rk2 || !back || !var<VAR_FORWARD>("forward", kTilesVar, g, n, sms) ||
                        !var<VAR_RECOMPUTE>("recompute", kTilesVar, g, n, sms) ||
                        !var<VAR_LAMBDA>("lambda", kTilesAdj, g, n, sms) || !var<VAR_MU>("mu", kTilesAdj, g, n, sms))
                        return 1;
                }
                const int hs = march_rows(gs, sms);
                if (hs < 1 || hs > nx) {
                    printf("strips of %d of %d rows\n", hs, nx);
                    return 1;
                }
            }
    printf("ok\n");
    return 0;
}
