// Host-side check of how heat runs are cut into overlapped blocks
// (heat_block.cuh): for grids of every size and run length, each launch that a
// plan leads to has a tile with exact rows and columns left, whole lanes of
// halo, and no more warps than its kernel allows; the streams' strips cover the
// rows.  Built and run by tests/test_host_block_plan.py (nvcc, no GPU needed).
#include <cstdio>

#include "../../pysweep_b200/csrc/heat_block.cuh"

using namespace psb;

template <int N>
int check(const TileShape (&shapes)[N], int step, int sms)
{
    for (int nx : {4, 8, 24, 50, 112, 160, 250, 481, 1120, 2048, 5000, 8192, 30000})
        for (int ny : {4, 8, 30, 112, 160, 390, 1000, 2048, 8192, 20000})
            for (int n : {1, 2, 3, 7, 8, 9, 15, 16, 17, 100, 5000})
                for (int maxT : {step, 3, 8, 16}) {
                    const int nl = n - n % step;
                    if (nl < step || maxT < step) continue;
                    const BlockGrid one{nx, ny};
                    const BlockGrids g{&one, 1};
                    const BlockPlan p = plan_block(shapes, g, nl, step, maxT, sms);
                    if (p.T < step || p.T % step || p.T > kTileMaxT || (p.T > maxT && maxT % step == 0) ||
                        (p.stream && (p.T != kStreamT || maxT < kStreamT))) {
                        printf("plan %dx%d n %d maxT %d: T %d\n", nx, ny, nl, maxT, p.T);
                        return 1;
                    }
                    for (int T = step; T <= p.T; T += step) {
                        double us;
                        const TileShape t = best_tile(shapes, T, g, sms, &us);
                        const int halo = (32 * t.C - tile_vw(t, T)) / 2;
                        if (tile_vh(t, T) < 2 || tile_vw(t, T) < 8 || halo < T || halo % t.C ||
                            t.nw > t.maxw || !(us < 1e300)) {
                            printf("tile %dx%d T %d\n", nx, ny, T);
                            return 1;
                        }
                    }
                    const int rows = stream_rows(g, sms);
                    if (rows < 1 || rows > nx) {
                        printf("strip rows %d of %d\n", rows, nx);
                        return 1;
                    }
                }
    return 0;
}

int main()
{
    for (int sms : {1, 16, 132, 148})
        if (check(kTilesFE, 1, sms) || check(kTilesRK2, 2, sms)) return 1;
    printf("ok\n");
    return 0;
}
