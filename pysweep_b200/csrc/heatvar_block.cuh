// Overlapped space-time tiles with a courant number per cell: the
// differentiable heat solve's forward steps, the recompute of a checkpoint
// segment and its adjoint steps, up to kTileMaxT levels per launch.
//
// The tiles of heat_block.cuh (nw warps x R rows x 32 C columns in registers,
// outer rows exchanged through shared memory every level), with the courant
// numbers in registers beside them (in shared memory their loads took more of
// the LSU than the levels of the FP64 pipe: forward at 2048², 6.5 -> 5.1 us per
// level).  The Laplacians that the recompute stores and the adjoint reads are
// touched at the exact cells only, once per level; in the adjoint each row's are
// loaded a level ahead.  Every cell sees the operations of single steps in
// their order, so the levels per launch change no bit.
//
// What bounds them: 8 or 9 FP64 operations per cell and level, for the
// recompute and the adjoint 8 bytes of Laplacian per cell and level each, and
// the start and end of every tile, which few warps per SM leave uncovered.
// (us per level, forward / recompute / adjoint: 512² 0.63 / 0.96 / 0.98,
// 1024 x 1536 2.2 / 3.5 / 5.1, 2048² 5.1 / 9.3 / 14.8; one and two levels per
// launch before: 2048² 15.3 / 36.8 together.)
#pragma once
#include "heat_block.cuh"
#include "launch.cuh"

namespace psb {

enum VarRole {
    VAR_FORWARD = 0,    // u' = (C dxx + C dyy) + u
    VAR_RECOMPUTE = 1,  // the same, storing every old level's dxx + dyy
    VAR_LAMBDA = 2,     // l' = l + L(C l), g += l L(u)
    VAR_MU = 3          // mu' as u', g += mu L(u)
};

struct VarArgs {
    const double* in;
    double* out;      // null: only the Laplacians are wanted (recompute)
    const double* C;
    double* lap;      // Laplacians of level 1 of the launch ...
    long long step;   // ... and the elements from one level's to the next's
    double* g;        // sums, updated in place
    int nx, ny, T, ncs, vw, vh;
};

// One row: old rows U, M, N (above, at, below) -> new row o and the old
// Laplacian l; the lateral neighbours from the adjacent lanes.
template <int C>
__device__ __forceinline__ void var_row(const double (&U)[C], const double (&M)[C],
                                        const double (&N)[C], const double (&cr)[C],
                                        double (&o)[C], double (&l)[C])
{
    const double left = __shfl_up_sync(0xffffffffu, M[C - 1], 1);
    const double right = __shfl_down_sync(0xffffffffu, M[0], 1);
    double t[C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
        const double c = M[j];
        const double ym = j == 0 ? left : M[j - 1], yp = j == C - 1 ? right : M[j + 1];
        const double rx = __dadd_rn(__fma_rn(-2.0, c, N[j]), U[j]);
        const double ry = __dadd_rn(__fma_rn(-2.0, c, yp), ym);
        t[j] = __dadd_rn(__dadd_rn(__dmul_rn(cr[j], rx), __dmul_rn(cr[j], ry)), c);
        l[j] = __dadd_rn(rx, ry);
    }
#pragma unroll
    for (int j = 0; j < C; ++j) o[j] = t[j];
}

// two columns of a field; ODD: one by one (a field 8 bytes off a 16-byte boundary)
template <bool ODD>
__device__ __forceinline__ double2 ld_two(const double* p)
{
    return ODD ? make_double2(p[0], p[1]) : *reinterpret_cast<const double2*>(p);
}

// ODD: some field of a solver is not 16-byte aligned (2048², us per level of
// forward, mu, lambda, aligned / odd: 5.6 / 6.1, 17.4 / 17.6, 19.0 / 19.8; the
// shared-memory prisms 33, 49, 84).
template <int ROLE, int C, int R, int MAXW, bool ODD>
__global__ void __launch_bounds__(32 * MAXW, 1) heatvar_tile(const __grid_constant__ VarArgs a)
{
    extern __shared__ __align__(16) double tile_sm[];
    constexpr bool ADJ = ROLE >= VAR_LAMBDA;
    constexpr int NP = C / 2;
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nx = a.nx, ny = a.ny, T = a.T;
    const int cs = blockIdx.x % a.ncs, rs = blockIdx.x / a.ncs;
    const int rlo = rs * a.vh, rhi = min(rlo + a.vh, nx);  // exact rows
    const int clo = cs * a.vw, chi = min(clo + a.vw, ny);  // exact columns
    const int c0 = clo - tile_halo<C>(T) + C * lane;
    const int r0 = rlo - T + w * R;
    int gp[NP];
    bool ok[NP];  // the pair's cells are exact
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int c = c0 + 2 * p;
        gp[p] = wrap(c, ny);
        ok[p] = c >= clo && c < chi;
    }
    auto mine = [&](int i) { return r0 + i >= rlo && r0 + i < rhi; };
    // level m's Laplacians of row i, at the exact cells
    auto load_lap = [&](int m, int i, double (&v)[C]) {
        if (m <= T && mine(i)) {
            const double* src = a.lap + (m - 1) * a.step + (size_t)(r0 + i) * ny + c0;
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (ok[p]) {
                    const double2 x = ODD ? make_double2(__ldcs(src + 2 * p), __ldcs(src + 2 * p + 1))
                                          : __ldcs(reinterpret_cast<const double2*>(src + 2 * p));
                    v[2 * p] = x.x;
                    v[2 * p + 1] = x.y;
                }
        }
    };
    // u[1..R]: the warp's rows (the forward levels move them to u[0..R-1] and
    // back)
    double u[R + 1][C], cr[R][C], g[ADJ ? R : 1][C], lp[ADJ ? R : 1][C];
    grid_wait();
    {
        int r = wrap(r0, nx);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const size_t o = (size_t)r * ny;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                const double2 v = ld_two<ODD>(a.in + o + gp[p]);
                const double2 c = ld_two<ODD>(a.C + o + gp[p]);
                u[i + 1][2 * p] = v.x;
                u[i + 1][2 * p + 1] = v.y;
                cr[i][2 * p] = c.x;
                cr[i][2 * p + 1] = c.y;
            }
            r = r + 1 == nx ? 0 : r + 1;
        }
        if constexpr (ADJ) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
#pragma unroll
                for (int j = 0; j < C; ++j) lp[i][j] = 0.0;
                load_lap(1, i, lp[i]);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    double2 v = make_double2(0.0, 0.0);
                    if (mine(i) && ok[p]) v = ld_two<ODD>(a.g + (size_t)(r0 + i) * ny + c0 + 2 * p);
                    g[i][2 * p] = v.x;
                    g[i][2 * p + 1] = v.y;
                }
            }
        }
    }
    grid_release();
    auto slot = [&](int buf, int ww, int b) {
        return tile_sm + ((buf * nw + ww) * 2 + b) * (32 * C) + lane * 2;
    };
    auto put = [&](int buf, int b, const double (&v)[C]) {
        double* q = slot(buf, w, b);
#pragma unroll
        for (int p = 0; p < NP; ++p)
            *reinterpret_cast<double2*>(q + p * 64) = make_double2(v[2 * p], v[2 * p + 1]);
    };
    auto get = [&](int buf, int ww, int b, double (&v)[C]) {
        const double* q = slot(buf, ww, b);
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const double2 x = *reinterpret_cast<const double2*>(q + p * 64);
            v[2 * p] = x.x;
            v[2 * p + 1] = x.y;
        }
    };
    auto store_row = [&](double* dst, int i, const double (&v)[C]) {
        if (!mine(i)) return;
        double* row = dst + (size_t)(r0 + i) * ny;
        if constexpr (ODD) {
#pragma unroll
            for (int j = 0; j < C; ++j)
                if (ok[j / 2]) row[c0 + j] = v[j];
        } else {
            block_store<C, double>(row, c0, clo, chi, 0, v);
        }
    };
    const int wu = w == 0 ? 0 : w - 1, wd = w == nw - 1 ? w : w + 1;
    double l[C];
    if constexpr (ADJ) {
        // rows in ascending order at every level: a row's Laplacians of the
        // next level have a whole level to arrive.  Exchanged, and differenced:
        // mu, or C .* lambda
        auto operand = [&](int i, double (&m)[C]) {
#pragma unroll
            for (int j = 0; j < C; ++j)
                m[j] = ROLE == VAR_LAMBDA ? __dmul_rn(cr[i][j], u[i + 1][j]) : u[i + 1][j];
        };
        double m0[C], m1[C], m2[C];
        operand(0, m0);
        put(0, 0, m0);
        operand(R - 1, m0);
        put(0, 1, m0);
        __syncthreads();
        for (int m = 1; m <= T; ++m) {
            const int b = (m - 1) & 1;
            get(b, wu, 1, m0);
            operand(0, m1);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if (i < R - 1) operand(i + 1, m2);
                else get(b, wd, 0, m2);
                // the sums, and the row's Laplacians of the next level
#pragma unroll
                for (int j = 0; j < C; ++j) g[i][j] = __fma_rn(u[i + 1][j], lp[i][j], g[i][j]);
                load_lap(m + 1, i, lp[i]);
                if constexpr (ROLE == VAR_MU) {
                    var_row<C>(m0, m1, m2, cr[i], u[i + 1], l);
                } else {
                    const double left = __shfl_up_sync(0xffffffffu, m1[C - 1], 1);
                    const double right = __shfl_down_sync(0xffffffffu, m1[0], 1);
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        const double c = m1[j];
                        const double ym = j == 0 ? left : m1[j - 1], yp = j == C - 1 ? right : m1[j + 1];
                        const double lm = __dadd_rn(__dadd_rn(__fma_rn(-2.0, c, m2[j]), m0[j]),
                                                    __dadd_rn(__fma_rn(-2.0, c, yp), ym));
                        u[i + 1][j] = __dadd_rn(u[i + 1][j], lm);
                    }
                }
                if (i == 0 || i == R - 1) {
                    double q[C];
                    operand(i, q);
                    put(1 - b, i == 0 ? 0 : 1, q);
                }
#pragma unroll
                for (int j = 0; j < C; ++j) {
                    m0[j] = m1[j];
                    m1[j] = m2[j];
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            store_row(a.out, i, u[i + 1]);
            store_row(a.g, i, g[i]);
        }
    } else {
        put(0, 0, u[1]);
        put(0, 1, u[R]);
        __syncthreads();
        double up[C], dn[C], last[C];
        // row i of level m from old rows A, B, D into o
        auto row = [&](int m, int i, const double (&A)[C], const double (&B)[C], const double (&D)[C],
                       double (&o)[C]) {
            var_row<C>(A, B, D, cr[i], o, l);
            if (ROLE == VAR_RECOMPUTE) store_row(a.lap + (m - 1) * a.step, i, l);
        };
        auto finish = [&](int k) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                if (a.out) store_row(a.out, i, u[i + k]);
            }
        };
        int m = 1;
        for (;;) {
            // u[1..R] -> u[0..R-1]: the outer rows first, for the neighbours
            get(0, wu, 1, up);
            get(0, wd, 0, dn);
            row(m, 0, up, u[1], u[2], u[0]);
            put(1, 0, u[0]);
            row(m, R - 1, u[R - 1], u[R], dn, last);
            put(1, 1, last);
#pragma unroll
            for (int i = 1; i < R - 1; ++i) {
                row(m, i, u[i], u[i + 1], u[i + 2], u[i]);
                }
#pragma unroll
            for (int j = 0; j < C; ++j) u[R - 1][j] = last[j];
            if (m++ == T) {
                finish(0);
                return;
            }
            __syncthreads();
            // u[0..R-1] -> u[1..R]
            get(1, wu, 1, up);
            get(1, wd, 0, dn);
            row(m, R - 1, u[R - 2], u[R - 1], dn, u[R]);
            put(0, 1, u[R]);
            row(m, 0, up, u[0], u[1], last);
            put(0, 0, last);
#pragma unroll
            for (int i = R - 2; i > 0; --i) {
                row(m, i, u[i - 1], u[i], u[i + 1], u[i + 1]);
                }
#pragma unroll
            for (int j = 0; j < C; ++j) u[1][j] = last[j];
            if (m++ == T) {
                finish(1);
                return;
            }
            __syncthreads();
        }
    }
}

// --------------------------------------------------------------- launches --
// (eight rows of state and courant numbers leave registers for 16 warps on an
// SM; six rows with the adjoint's sums and Laplacians beside them, too)
constexpr TileShape kTilesVar[] = {{2, 8, 16, 16}, {2, 8, 12, 16}, {2, 8, 8, 16}, {2, 8, 4, 16},
                                   {2, 4, 12, 24}, {2, 4, 8, 24},  {2, 4, 6, 24}};
constexpr TileShape kTilesAdj[] = {{2, 6, 16, 16}, {2, 6, 12, 16}, {2, 6, 8, 16}, {2, 6, 6, 16},
                                   {2, 6, 4, 16},  {2, 4, 10, 20}, {2, 4, 6, 20}};

// Relative cost of the roles' tiles, fitted to launches of 256² to 2048²:
// the Laplacians' stores, and in the adjoint their loads and the sums.
template <int ROLE>
constexpr TileCost var_cost()
{
    return ROLE == VAR_FORWARD ? TileCost{1.0, 1.5, 1.5, 1.0}
                               : (ROLE == VAR_RECOMPUTE ? TileCost{1.8, 2.0, 1.5, 1.0} : TileCost{1.6, 3.0, 1.5, 1.0});
}

template <int ROLE>
BlockPlan plan_var(const BlockGrids& g, int nlevels, int sms)
{
    if constexpr (ROLE >= VAR_LAMBDA)
        return plan_tiles(kTilesAdj, g, nlevels, 1, kTileMaxT, sms, var_cost<ROLE>());
    else
        return plan_tiles(kTilesVar, g, nlevels, 1, kTileMaxT, sms, var_cost<ROLE>());
}

// One launch of T levels; a: pointers, nx, ny.
template <int ROLE, bool ODD = false>
void launch_var(VarArgs a, int T, int sms, cudaStream_t st)
{
    constexpr bool ADJ = ROLE >= VAR_LAMBDA;
    const BlockGrid grid{a.nx, a.ny};
    const BlockGrids g{&grid, 1};
    double us;
    TileShape t;
    if constexpr (ADJ) t = best_tile(kTilesAdj, T, g, sms, &us, var_cost<ROLE>());
    else t = best_tile(kTilesVar, T, g, sms, &us, var_cost<ROLE>());
    a.T = T;
    a.vw = tile_vw(t, T);
    a.vh = tile_vh(t, T);
    a.ncs = (a.ny + a.vw - 1) / a.vw;
    const int units = a.ncs * ((a.nx + a.vh - 1) / a.vh);
    const size_t smem = tile_smem<2>(t.nw);
    if (t.R == 4)
        launch_after(heatvar_tile<ROLE, 2, 4, ADJ ? 20 : 24, ODD>, units, 32 * t.nw, smem, st, a);
    else
        launch_after(heatvar_tile<ROLE, 2, ADJ ? 6 : 8, 16, ODD>, units, 32 * t.nw, smem, st, a);
}

// --------------------------------------------------------------- backward --
// T levels of a checkpoint segment backward in one launch: a tile steps the
// state the levels start from forward once more, keeping its exact cells'
// Laplacians in shared memory, then lambda backward through them, so that they
// never reach global memory.
//
// What bounds it: the two passes one after the other, 17 FP64 operations per
// cell and level on cells of which a quarter is halo, and 48 bytes per cell and
// launch; at most 227 KB of Laplacians on an SM.  Two CTAs or more per SM: with
// one, its loads and stores hide behind nothing (2048², T = 4, 8 warps of 6 rows
// twice 14.4, 16 warps once 21.9 us per level).  us per level, recompute +
// adjoint by themselves / here with the forward steps that lead to the levels'
// start: 256² 2.08 / 1.50, 512² 2.67 / 2.24, 1024 x 1536 9.4 / 8.25, 2048² 26.6 / 20.1,
// 4096² 96 / 75.
struct BackArgs {
    const double* u;    // the state before the levels
    const double* C;
    const double* in;   // lambda after them
    double* out;        // and before them
    double* g;          // sums, updated in place
    int nx, ny, T, ncs, vw, vh;
};

// Shared memory: the outer rows, then Laplacians [level][exact row][lane][2].
__host__ __device__ constexpr size_t back_smem(int R, int nw, int T)
{
    return tile_smem<2>(nw) + sizeof(double) * 64 * T * (nw * R - 2 * T);
}

// MAXW warps per CTA, two such CTAs on an SM.
template <int R, int MAXW>
__global__ void __launch_bounds__(32 * MAXW, 2) heatvar_back(const __grid_constant__ BackArgs a)
{
    extern __shared__ __align__(16) double tile_sm[];
    constexpr int C = 2;
    const int nw = blockDim.x >> 5, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nx = a.nx, ny = a.ny, T = a.T;
    const int cs = blockIdx.x % a.ncs, rs = blockIdx.x / a.ncs;
    const int rlo = rs * a.vh, rhi = min(rlo + a.vh, nx);  // exact rows
    const int clo = cs * a.vw, chi = min(clo + a.vw, ny);  // exact columns
    const int c0 = clo - tile_halo<C>(T) + C * lane;
    const int r0 = rlo - T + w * R;
    const int gcol = wrap(c0, ny);
    const bool ok = c0 >= clo && c0 < chi;
    const int ne = nw * R - 2 * T;  // exact rows of a whole tile
    double* lap = tile_sm + 32 * C * nw * 4 + lane * 2;
    // where level m's Laplacian of the warp's row i lies; rows that are exact
    auto lap_at = [&](int m, int i) { return lap + ((m - 1) * ne + w * R + i - T) * 64; };
    auto kept = [&](int i) { return w * R + i >= T && w * R + i < T + ne; };
    auto mine = [&](int i) { return r0 + i >= rlo && r0 + i < rhi && ok; };
    auto slot = [&](int buf, int ww, int b) {
        return tile_sm + ((buf * nw + ww) * 2 + b) * (32 * C) + lane * 2;
    };
    auto put = [&](int buf, int b, const double (&v)[C]) {
        *reinterpret_cast<double2*>(slot(buf, w, b)) = make_double2(v[0], v[1]);
    };
    auto get = [&](int buf, int ww, int b, double (&v)[C]) {
        const double2 x = *reinterpret_cast<const double2*>(slot(buf, ww, b));
        v[0] = x.x;
        v[1] = x.y;
    };
    auto load = [&](const double* p, double (&v)[C]) {
        const double2 x = *reinterpret_cast<const double2*>(p);
        v[0] = x.x;
        v[1] = x.y;
    };
    const int wu = w == 0 ? 0 : w - 1, wd = w == nw - 1 ? w : w + 1;
    double cr[R][C], u[R][C], m0[C], m1[C], m2[C], l[C];
    grid_wait();
    {
        int r = wrap(r0, nx);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const size_t o = (size_t)r * ny + gcol;
            load(a.u + o, u[i]);
            load(a.C + o, cr[i]);
            r = r + 1 == nx ? 0 : r + 1;
        }
    }
    grid_release();
    put(0, 0, u[0]);
    put(0, 1, u[R - 1]);
    __syncthreads();
    // the states u_n .. : rows in ascending order, the old row above kept aside
    for (int m = 1; m <= T; ++m) {
        const int b = (m - 1) & 1;
        get(b, wu, 1, m0);
        get(b, wd, 0, m2);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            double old[C];
#pragma unroll
            for (int j = 0; j < C; ++j) old[j] = u[i][j];
            if (i < R - 1) var_row<C>(m0, old, u[i + 1], cr[i], u[i], l);
            else var_row<C>(m0, old, m2, cr[i], u[i], l);
            if (kept(i)) *reinterpret_cast<double2*>(lap_at(m, i)) = make_double2(l[0], l[1]);
#pragma unroll
            for (int j = 0; j < C; ++j) m0[j] = old[j];
            if (i == 0) put(1 - b, 0, u[0]);
        }
        put(1 - b, 1, u[R - 1]);
        __syncthreads();
    }
    // lambda backward: u now holds it
    double g[R][C];
    {
        int r = wrap(r0, nx);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const size_t o = (size_t)r * ny + gcol;
            load(a.in + o, u[i]);
            g[i][0] = g[i][1] = 0.0;
            if (mine(i)) load(a.g + (size_t)(r0 + i) * ny + c0, g[i]);
            r = r + 1 == nx ? 0 : r + 1;
        }
    }
    // exchanged, and differenced
    auto operand = [&](int i, double (&m)[C]) {
#pragma unroll
        for (int j = 0; j < C; ++j) m[j] = __dmul_rn(cr[i][j], u[i][j]);
    };
    operand(0, m0);
    put(0, 0, m0);
    operand(R - 1, m0);
    put(0, 1, m0);
    __syncthreads();
    for (int m = T; m >= 1; --m) {
        const int b = (T - m) & 1;
        get(b, wu, 1, m0);
        operand(0, m1);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (i < R - 1) operand(i + 1, m2);
            else get(b, wd, 0, m2);
            // (rows that are not exact take another row's: their sums go nowhere;
            // without the branch the rows overlap: 2048² 15.2 -> 14.4)
            load(lap + ((m - 1) * ne + min(max(w * R + i - T, 0), ne - 1)) * 64, l);
#pragma unroll
            for (int j = 0; j < C; ++j) g[i][j] = __fma_rn(u[i][j], l[j], g[i][j]);
            const double left = __shfl_up_sync(0xffffffffu, m1[1], 1);
            const double right = __shfl_down_sync(0xffffffffu, m1[0], 1);
            const double ym[C] = {left, m1[0]}, yp[C] = {m1[1], right};
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const double lm = __dadd_rn(__dadd_rn(__fma_rn(-2.0, m1[j], m2[j]), m0[j]),
                                            __dadd_rn(__fma_rn(-2.0, m1[j], yp[j]), ym[j]));
                u[i][j] = __dadd_rn(u[i][j], lm);
            }
            if (i == 0 || i == R - 1) {
                double q[C];
                operand(i, q);
                put(1 - b, i == 0 ? 0 : 1, q);
            }
#pragma unroll
            for (int j = 0; j < C; ++j) {
                m0[j] = m1[j];
                m1[j] = m2[j];
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (mine(i)) {
            const size_t o = (size_t)(r0 + i) * ny + c0;
            *reinterpret_cast<double2*>(a.out + o) = make_double2(u[i][0], u[i][1]);
            *reinterpret_cast<double2*>(a.g + o) = make_double2(g[i][0], g[i][1]);
        }
}

// The tiles that are built: six rows per warp and 8 warps twice on an SM, four
// rows and 10 warps.
constexpr int kBackMaxT = 8;
constexpr TileShape kTilesBack[] = {{2, 6, 8, 8}, {2, 6, 6, 8}, {2, 6, 4, 8},
                                    {2, 4, 10, 10}, {2, 4, 8, 10}};

// Estimated microseconds of one launch (fitted to launches of 256² to 2048²,
// within 30%), or 0 where no cell of the tile stays exact.
inline double back_us(const TileShape& t, int T, const BlockGrids& g, int sms)
{
    const int vw = tile_vw(t, T), vh = tile_vh(t, T);
    if (vw < 8 || vh < 2) return 0.0;
    const int occ = std::min(2 * t.maxw / t.nw, (int)(227 * 1024 / (back_smem(t.R, t.nw, T) + 1024)));
    if (occ < 1) return 0.0;
    const double n = (double)((g.blocks(vw, vh) + sms - 1) / sms), rounds = std::max(1.0, n / occ);
    return 1.24 + n * (0.0061 * T + 0.04) * t.nw * t.R + (0.39 * T + 0.38) * rounds;
}

inline TileShape best_back(int T, const BlockGrids& g, int sms, double* us)
{
    TileShape best = kTilesBack[0];
    *us = 1e300;
    for (const TileShape& t : kTilesBack) {
        const double one = back_us(t, T, g, sms);
        if (one > 0 && one < *us) {
            *us = one;
            best = t;
        }
    }
    return best;
}

inline BlockPlan plan_back(const BlockGrids& g, int nlevels, int sms)
{
    BlockPlan best{false, 1, 1e300};
    for (int T = 1; T <= kBackMaxT; ++T) {
        const int k = (nlevels + T - 1) / T;
        double one;
        best_back(T, g, sms, &one);
        if (k * one < best.us) best = BlockPlan{false, T, k * one};
    }
    return best;
}

// One launch of T levels; a: pointers, nx, ny.
inline void launch_back(BackArgs a, int T, int sms, cudaStream_t st)
{
    const BlockGrid grid{a.nx, a.ny};
    double us;
    const TileShape t = best_back(T, BlockGrids{&grid, 1}, sms, &us);
    a.T = T;
    a.vw = tile_vw(t, T);
    a.vh = tile_vh(t, T);
    a.ncs = (a.ny + a.vw - 1) / a.vw;
    const int units = a.ncs * ((a.nx + a.vh - 1) / a.vh);
    const size_t smem = back_smem(t.R, t.nw, T);
    auto k = t.R == 6 ? heatvar_back<6, 8> : heatvar_back<4, 10>;
    allow_big_smem(k);
    launch_after(k, units, 32 * t.nw, smem, st, a);
}

}  // namespace psb
