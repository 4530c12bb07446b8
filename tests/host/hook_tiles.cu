// Host-side check of the step hooks' tiles (hook.cuh): for every number of
// variables and every reach, the tile fits, keeps exact cells, and a launch of one
// level leaves an SM the warps it can have: 16 rows' worth, or all that any tile
// fits.  Built and run by tests/test_host_hook_tiles.py (nvcc, no GPU needed).
#include <cstdio>

#include "../../pysweep_b200/csrc/hook.cuh"

using namespace psb;

// warps of a launch of one level on an SM: its CTAs, a warp to a row at most
static int warps(int nv, int ops, int rows, int threads)
{
    const size_t sm = hook_block_smem(nv, ops, rows, 1);
    if (sm > 227 * 1024) return 0;
    const int ctas = (int)(228 * 1024 / (sm + 1024));
    return std::min(ctas, 2048 / threads) * std::min(rows, threads / 32);
}

int main()
{
    for (int nv = 1; nv <= 8; ++nv)
        for (int ops = 1; ops <= 4; ++ops)
        for (const long long cells : {256LL, 512LL * 512, 1LL << 26}) {
            for (int maxT = 1; maxT <= kHookBlkMaxT; ++maxT) {
                const HookBlock b = hook_block(nv, ops, maxT, cells, 148);
                const int ih = b.rows - 2 * ops * (b.T - 1), iw = kHookBlkW - 2 * ops * (b.T - 1);
                if (b.rows < 1 || b.T < 1 || b.T > maxT || ih < 1 || iw < 2 || iw % 2 ||
                    hook_block_smem(nv, ops, b.rows, b.T) > 227 * 1024) {
                    printf("nv %d ops %d maxT %d: rows %d T %d\n", nv, ops, maxT, b.rows, b.T);
                    return 1;
                }
            }
            const HookBlock b = hook_block(nv, ops, 1, cells, 148);
            int most = 0;
            for (int rows : {32, 16, 8, 4})
                for (int threads : {kHookBlkNT / 2, kHookBlkNT}) most = std::max(most, warps(nv, ops, rows, threads));
            const int have = warps(nv, ops, b.rows, b.threads1);
            if (have < std::min(most, 16)) {
                printf("nv %d ops %d: %d rows, %d threads: %d warps of %d\n", nv, ops, b.rows, b.threads1,
                       have, most);
                return 1;
            }
        }
    printf("ok\n");
    return 0;
}
