// Overlapped space-time blocks for the heat equation: several levels per
// launch, every block complete by itself.
//
// A block reads its cells and a halo of one cell per level, advances T levels
// on chip and writes the cells that are still exact.  Neighbouring blocks
// evaluate the cells of their common halo twice, by the same per-cell function,
// so the result is that of the prism / bridge / gap decomposition and of the
// standard one, bit for bit, and nothing but the field passes between blocks:
// no faces, no seams, one launch per T levels.
//
// What bounds it: eight FP64 operations per cell and level on a pipe that
// takes two cycles per warp and operation (148 SMs x 64 lanes at 1965 MHz:
// 2327 G cells/s), less the cells evaluated twice.  Two kernels, by size:
//
//   heat_block_stream  One warp streams a strip of 128 columns down its rows
//       with T = 8 levels in flight, all state in registers: lane l holds
//       columns 4l .. 4l+3 and three rows of every level (above, centre,
//       below, rotating by name over three unrolled steps: no moves).  A step
//       takes one new row and computes one row of every level.  The levels
//       run in groups of two, each group one row behind the one before it, so
//       a step holds four independent chains instead of one of eight (8192²:
//       346 -> 329 us per 8 levels, the kernel alone; 339 in a run's row of
//       launches, 367 once a long one has met the 1000 W cap).  112 of the 128
//       columns are exact at the end (12.5% evaluated twice).
//   heat_block_tile    A CTA holds a tile of nw x R rows and 32 C columns in
//       registers and steps it in place, neighbouring warps exchanging one
//       row each way per level through shared memory.  Rows of a warp are
//       independent, so two warps per scheduler fill the FP64 pipe; the halo
//       is paid in both directions.  Used where the rows are too few for
//       strips (a strip's 2 T rows of run-in weigh more than the tile's), for
//       the levels left over by T = 8 and for levels kept as frames.
//
// Global traffic per cell and 8 levels: one read (1.14x) and one write, 2.0
// bytes per cell and level.
#pragma once
#include <algorithm>
#include <type_traits>

#include "heat_cell.cuh"
#include "launch.cuh"

namespace psb {

constexpr int kStreamT = 8;    // levels per launch of the streams
constexpr int kTileMaxT = 16;  // most levels per launch of the tiles
constexpr int kBlockRing = 4;  // rows of a stream in flight (cp.async)

struct BlockArgs {
    const void* in;  // the newest level
    void* out;       // T levels on
    void* out1;      // two-stage scheme: the level before it, when kept
    int nx, ny;
    int T;         // levels of this launch (tiles)
    int ncs;       // column strips
    int vw, vh;    // exact columns / rows of a block
    int units;     // blocks
    int v4;        // rows are whole groups of four columns: 4-wide accesses
    int nframe;    // levels kept as frames in this launch
    double cr;
    void* frame[kTileMaxT];  // frame of level m+1, or null
};

// the grid this one depends on has finished and its writes are visible
// (programmatic dependent launch; returns at once without one)
__device__ __forceinline__ void grid_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// the next grid of the stream may take up the SMs this one leaves
__device__ __forceinline__ void grid_release()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// four consecutive columns at once (32 bytes of double, 16 of float); stores
// half this wide left every 32-byte sector to be merged in L2 (8192²: 375 ->
// 357 us per 8 levels)
__device__ __forceinline__ void st_quad(double* p, const double* v)
{
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
                 "d"(v[2]), "d"(v[3])
                 : "memory");
}
__device__ __forceinline__ void st_quad(float* p, const double* v)
{
    *reinterpret_cast<float4*>(p) =
        make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
}
__device__ __forceinline__ void ld_quad(const double* p, double* v)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void ld_quad(const float* p, double* v)
{
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x;
    v[1] = x.y;
    v[2] = x.z;
    v[3] = x.w;
}

// C columns of one row from the rows above, at and below (U, M, N), the outer
// columns' neighbours from the adjacent lanes.  KIND 0: a forward Euler level.
// KIND 1: the half stage.  KIND 2: the full stage, from the level before the
// half stage (B).  Lanes 0 and 31 take their own values where they have no
// neighbour: those cells lie in the halo.
template <int KIND, int C, class S>
__device__ __forceinline__ void block_row(const double (&U)[C], const double (&M)[C],
                                          const double (&N)[C], const double (&B)[C],
                                          double (&o)[C], double cr)
{
    const double left = __shfl_up_sync(0xffffffffu, M[C - 1], 1);
    const double right = __shfl_down_sync(0xffffffffu, M[0], 1);
    double t[C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
        const double c = M[j];
        const double ym = j == 0 ? left : M[j - 1], yp = j == C - 1 ? right : M[j + 1];
        if constexpr (KIND == 0) {
            t[j] = to_level<S>(heat_fe(c, U[j], N[j], ym, yp, cr));
        } else {
            const double dxx = __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, c, N[j]), U[j]));
            const double dyy = __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, c, yp), ym));
            const double cd = __dadd_rn(dxx, dyy);
            // heat.py:53-57: coeff * cd + base, coeff 0.5 or 1
            t[j] = KIND == 1 ? __dadd_rn(__dmul_rn(0.5, cd), c) : __dadd_rn(cd, B[j]);
        }
    }
#pragma unroll
    for (int j = 0; j < C; ++j) o[j] = t[j];
}

// exact rows and columns of one row -> global
template <int C, class S>
__device__ __forceinline__ void block_store(S* row, int c0, int clo, int chi, int v4,
                                            const double (&v)[C])
{
    using P = typename Pair2<S>::type;
    if (C == 4 && v4) {
        if (c0 >= clo && c0 < chi) st_quad(row + c0, v);
    } else {
#pragma unroll
        for (int p = 0; p < C / 2; ++p) {
            const int c = c0 + 2 * p;
            if (c >= clo && c < chi)
                *reinterpret_cast<P*>(row + c) = pair2<S>(v[2 * p], v[2 * p + 1]);
        }
    }
}

// ---------------------------------------------------------------- streams --
// Exact columns of a strip.
constexpr int kStreamC = 4, kStreamW = 32 * kStreamC - 2 * kStreamT;

// One strip: columns [cs vw, +vw), rows [x0, x1).  RK2: the levels alternate
// half and full stage, starting with a half stage.
template <class S, bool RK2>
__device__ __forceinline__ void block_stream_body(const BlockArgs& a, int unit, S* ring)
{
    using P = typename Pair2<S>::type;
    constexpr int T = kStreamT, C = kStreamC, G = T / 2, VW = kStreamW;
    const int lane = threadIdx.x & 31;
    const int nx = a.nx, ny = a.ny;
    const int cs = unit % a.ncs, rs = unit / a.ncs;
    const int x0 = rs * a.vh, x1 = min(x0 + a.vh, nx);
    const int nin = x1 - x0 + 2 * T;  // rows read
    const int n = nin + G - 1;        // steps
    const int clo = cs * VW, chi = min(clo + VW, ny);
    const int c0 = clo - T + C * lane;  // this lane's first column
    const int g0 = wrap(c0, ny), g1 = wrap(c0 + 2, ny);
    const S* in = reinterpret_cast<const S*>(a.in);
    int ir = wrap(x0 - T, nx);
    auto issue = [&](int s) {  // row s of the strip starts arriving
        if (s < nin) {
            S* sl = ring + (s % kBlockRing) * (32 * C) + lane * 2;
            const S* row = in + (size_t)ir * ny;
            cp_async_pair<S>(sl, row + g0);
            cp_async_pair<S>(sl + 64, row + g1);
            ir = ir + 1 == nx ? 0 : ir + 1;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kBlockRing - 1; ++s) issue(s);
    const double cr = a.cr;
    S* out = reinterpret_cast<S*>(a.out) + (ptrdiff_t)(x0 - 2 * T - (G - 1)) * ny;

    // three rows of every level: level t's rows in X[t], Y[t], Z[t]
    double X[T][C], Y[T][C], Z[T][C];
#pragma unroll
    for (int t = 0; t < T; ++t)
#pragma unroll
        for (int j = 0; j < C; ++j) X[t][j] = Y[t][j] = Z[t][j] = 0.0;

    // Step s with the first NG groups: U, M, N hold the rows above, at and
    // below each level's new row.  The later groups go first: a group's last
    // row replaces the row above of the next group's first level, which that
    // group has just used for the last time, and is its row below one step on.
    auto step = [&](auto ng, int s, double (&U)[T][C], double (&M)[T][C], double (&N)[T][C]) {
        constexpr int NG = decltype(ng)::value;
        cp_async_wait<kBlockRing - 2>();
        const S* sl = ring + (s % kBlockRing) * (32 * C) + lane * 2;
        const double2 v0 = widen(*reinterpret_cast<const P*>(sl));
        const double2 v1 = widen(*reinterpret_cast<const P*>(sl + 64));
        N[0][0] = v0.x;
        N[0][1] = v0.y;
        N[0][2] = v1.x;
        N[0][3] = v1.y;
        issue(s + kBlockRing - 1);
        double o[C];
#pragma unroll
        for (int q = NG - 1; q >= 0; --q) {
            const int t = 2 * q;
            block_row<RK2 ? 1 : 0, C, S>(U[t], M[t], N[t], U[t], N[t + 1], cr);
            if (q == G - 1)
                block_row<RK2 ? 2 : 0, C, S>(U[t + 1], M[t + 1], N[t + 1], U[t], o, cr);
            else
                block_row<RK2 ? 2 : 0, C, S>(U[t + 1], M[t + 1], N[t + 1], U[t], U[t + 2], cr);
        }
        if (NG == G && s >= 2 * T + G - 1 && s < n)
            block_store<C, S>(out + (size_t)s * ny, c0, clo, chi, a.v4, o);
    };
    auto three = [&](auto ng, int s) {
        step(ng, s, X, Y, Z);
        step(ng, s + 1, Y, Z, X);
        step(ng, s + 2, Z, X, Y);
    };
    // Run-in: group q's first exact row comes at step 5 q + 2, so the later
    // groups join in turn.
    three(std::integral_constant<int, 1>(), 0);
    three(std::integral_constant<int, 2>(), 3);
    three(std::integral_constant<int, 2>(), 6);
    three(std::integral_constant<int, 3>(), 9);
    three(std::integral_constant<int, 3>(), 12);
    for (int s = 15; s < n; s += 3) three(std::integral_constant<int, G>(), s);
}

template <class S, bool RK2>
__global__ void __launch_bounds__(32, 8) heat_block_stream(const __grid_constant__ BlockArgs a)
{
    __shared__ __align__(16) S ring[kBlockRing * 32 * kStreamC];
    grid_wait();
    grid_release();
    block_stream_body<S, RK2>(a, blockIdx.x, ring);
}

// ------------------------------------------------------------------ tiles --
// Shared memory of a tile: two buffers of every warp's outer rows.
template <int C>
__host__ __device__ constexpr size_t tile_smem(int nw)
{
    return sizeof(double) * 2 * nw * 2 * 32 * C;
}
// Columns of halo on each side (whole lanes, so that the exact columns start
// at a lane).
template <int C>
__host__ __device__ constexpr int tile_halo(int T)
{
    return (T + C - 1) / C * C;
}

// One tile of nw warps x R rows by 32 C columns, a.T levels.
template <class S, bool RK2, int C, int R>
__device__ __forceinline__ void block_tile_body(const BlockArgs& a, int unit, int nw, double* sm)
{
    using P = typename Pair2<S>::type;
    constexpr int NP = C / 2;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nx = a.nx, ny = a.ny, T = a.T;
    const int cs = unit % a.ncs, rs = unit / a.ncs;
    const int rlo = rs * a.vh, rhi = min(rlo + a.vh, nx);  // exact rows
    const int clo = cs * a.vw, chi = min(clo + a.vw, ny);  // exact columns
    const int c0 = clo - tile_halo<C>(T) + C * lane;
    const int r0 = rlo - T + w * R;
    const double cr = a.cr;
    // u[1..R]: the warp's rows; a level moves them to u[0..R-1], the next one back
    double u[R + 1][C];
    {
        const S* in = reinterpret_cast<const S*>(a.in);
        int r = wrap(r0, nx);
        int g[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) g[p] = wrap(c0 + 2 * p, ny);
        if (C == 4 && a.v4) {
#pragma unroll
            for (int i = 1; i <= R; ++i) {
                ld_quad(in + (size_t)r * ny + g[0], u[i]);
                r = r + 1 == nx ? 0 : r + 1;
            }
        } else {
#pragma unroll
            for (int i = 1; i <= R; ++i) {
                const S* row = in + (size_t)r * ny;
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const double2 v = widen(*reinterpret_cast<const P*>(row + g[p]));
                    u[i][2 * p] = v.x;
                    u[i][2 * p + 1] = v.y;
                }
                r = r + 1 == nx ? 0 : r + 1;
            }
        }
    }
    grid_release();
    // outer rows, [buffer][warp][top, bottom][pair][lane][2]
    auto slot = [&](int buf, int ww, int b) {
        return sm + ((buf * nw + ww) * 2 + b) * (32 * C) + lane * 2;
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
    // the rows above the first and below the last warp are halo: any value does
    const int wu = w == 0 ? 0 : w - 1, wd = w == nw - 1 ? w : w + 1;
    auto store = [&](void* dst, const double (&v)[R + 1][C], int k) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = r0 + i;
            if (r >= rlo && r < rhi)
                block_store<C, S>(reinterpret_cast<S*>(dst) + (size_t)r * ny, c0, clo, chi, a.v4,
                                  v[i + k]);
        }
    };
    auto keep = [&](int m, const double (&v)[R + 1][C], int k) {  // frame of level m
        if (a.nframe && a.frame[m - 1]) store(a.frame[m - 1], v, k);
    };
    double up[C], dn[C];
    put(0, 0, u[1]);
    put(0, 1, u[R]);
    __syncthreads();
    if constexpr (!RK2) {
        double last[C];
        int m = 0;
        for (;;) {
            // u[1..R] -> u[0..R-1]: the outer rows first, for the neighbours
            get(0, wu, 1, up);
            get(0, wd, 0, dn);
            block_row<0, C, S>(up, u[1], u[2], up, u[0], cr);
            put(1, 0, u[0]);
            block_row<0, C, S>(u[R - 1], u[R], dn, up, last, cr);
            put(1, 1, last);
#pragma unroll
            for (int i = 1; i < R - 1; ++i) block_row<0, C, S>(u[i], u[i + 1], u[i + 2], up, u[i], cr);
#pragma unroll
            for (int j = 0; j < C; ++j) u[R - 1][j] = last[j];
            keep(++m, u, 0);
            if (m == T) {
                store(a.out, u, 0);
                return;
            }
            __syncthreads();
            // u[0..R-1] -> u[1..R]
            get(1, wu, 1, up);
            get(1, wd, 0, dn);
            block_row<0, C, S>(u[R - 2], u[R - 1], dn, up, u[R], cr);
            put(0, 1, u[R]);
            block_row<0, C, S>(up, u[0], u[1], up, last, cr);
            put(0, 0, last);
#pragma unroll
            for (int i = R - 2; i > 0; --i) block_row<0, C, S>(u[i - 1], u[i], u[i + 1], up, u[i + 1], cr);
#pragma unroll
            for (int j = 0; j < C; ++j) u[1][j] = last[j];
            keep(++m, u, 1);
            if (m == T) {
                store(a.out, u, 1);
                return;
            }
            __syncthreads();
        }
    } else {
        // T even: half stage into h, full stage back onto u
        double h[R + 1][C];
        for (int m = 2;; m += 2) {
            get(0, wu, 1, up);
            get(0, wd, 0, dn);
            block_row<1, C, S>(up, u[1], u[2], up, h[1], cr);
            put(1, 0, h[1]);
            block_row<1, C, S>(u[R - 1], u[R], dn, up, h[R], cr);
            put(1, 1, h[R]);
#pragma unroll
            for (int i = 2; i < R; ++i) block_row<1, C, S>(u[i - 1], u[i], u[i + 1], up, h[i], cr);
            keep(m - 1, h, 1);
            if (m == T && a.out1) store(a.out1, h, 1);
            __syncthreads();
            get(1, wu, 1, up);
            get(1, wd, 0, dn);
            block_row<2, C, S>(up, h[1], h[2], u[1], u[1], cr);
            put(0, 0, u[1]);
            block_row<2, C, S>(h[R - 1], h[R], dn, u[R], u[R], cr);
            put(0, 1, u[R]);
#pragma unroll
            for (int i = 2; i < R; ++i) block_row<2, C, S>(h[i - 1], h[i], h[i + 1], u[i], u[i], cr);
            keep(m, u, 1);
            if (m == T) {
                store(a.out, u, 1);
                return;
            }
            __syncthreads();
        }
    }
}

// MAXW warps per CTA and per SM (the register cap): a tile of nw warps leaves
// room for MAXW / nw on an SM.
template <class S, bool RK2, int C, int R, int MAXW>
__global__ void __launch_bounds__(32 * MAXW, 1) heat_block_tile(const __grid_constant__ BlockArgs a)
{
    extern __shared__ __align__(16) double tile_sm[];
    grid_wait();
    block_tile_body<S, RK2, C, R>(a, blockIdx.x, blockDim.x >> 5, tile_sm);
}

// ------------------------------------------------------------------- plan --
// The tiles that are built: C columns per lane, R rows per warp, nw warps,
// MAXW warps on an SM.
struct TileShape {
    int C, R, nw, maxw;
};

// (eight and ten rows of four columns: grids whose tiles then fit the SMs in
// fewer rounds, 1000 x 1400 1.73 -> 1.51 us per level, 1280² 1.95 -> 1.75)
constexpr TileShape kTilesFE[] = {{4, 6, 16, 16}, {4, 6, 12, 16}, {4, 6, 8, 16},  {4, 8, 16, 16},
                                  {4, 10, 12, 12}, {2, 8, 12, 20}, {2, 8, 8, 20},
                                  {2, 4, 12, 24}, {2, 4, 8, 24},  {2, 4, 6, 24},  {2, 4, 4, 24}};
// Two stages keep two fields in registers.  us per level with four rows of four
// columns and 16 warps, before / with these: 512² 0.95 / 0.60, 1120² 1.80 /
// 1.51, 1000 x 1400 1.95 / 1.84, 1536² 3.0 / 2.78.
constexpr TileShape kTilesRK2[] = {{4, 8, 12, 12}, {4, 6, 12, 12}, {4, 4, 16, 16},
                                   {2, 8, 16, 16}, {2, 8, 12, 16}, {2, 8, 8, 16},
                                   {2, 4, 12, 24}, {2, 4, 8, 24},  {2, 4, 6, 24}};

// How a run of levels is cut into launches: streams of kStreamT levels (and
// tiles for what is left), or tiles of at most T levels.
struct BlockPlan {
    bool stream;
    int T;
    double us;  // estimated time of the run
};

inline int tile_vw(const TileShape& t, int T) { return 32 * t.C - 2 * ((T + t.C - 1) / t.C * t.C); }
inline int tile_vh(const TileShape& t, int T) { return t.nw * t.R - 2 * T; }

// The grids of one launch: a solver's one, a batch's many.
struct BlockGrid {
    int nx, ny;
};
struct BlockGrids {
    const BlockGrid* g;
    int n;
    long long blocks(int vw, int vh) const
    {
        long long k = 0;
        for (int i = 0; i < n; ++i)
            k += (long long)((g[i].ny + vw - 1) / vw) * ((g[i].nx + vh - 1) / vh);
        return k;
    }
    int rows() const
    {
        int m = 1;
        for (int i = 0; i < n; ++i) m = std::max(m, g[i].nx);
        return m;
    }
};

// A tile's work relative to plain heat's: FP64 pipe time of a level, bytes of a
// tile, latency of a level.  two: a level of tiles of two columns and eight rows,
// whose warps exchange more per cell (1280²: 2.17 us per level where six rows of
// four columns take 1.96; without it they were planned at 1.95 and 1.98).
// four: one of tiles of four rows.  stream: a launch of the streams.
struct TileCost {
    double level = 1.0, bytes = 1.0, latency = 1.0, two = 1.1, four = 1.0, stream = 1.0;
};
// Two stages: fitted to launches of 160² to 2048² (the plan within 1% of the best
// tile there).
constexpr TileCost kCostRK2{1.0, 1.17, 1.0, 1.1, 1.15, 1.0};
// float32 fields: two conversions per cell and level, which the streams' warps
// hide better than a tile's (2048², float64 / float32, us per 8 levels: streams
// 32.2 / 36.6, tiles 36.4 / 46.7).
constexpr TileCost kCostF32{1.0, 1.0, 1.0, 1.1, 1.0, 0.91};

// Estimated microseconds of one launch of T levels in tiles of shape t, or 0
// where no cell of the tile stays exact.  Fitted to launches of 160² to 8192²
// (within 15%): a level of one tile takes its FP64 operations at the pipe's
// rate (16 cycles per warp and cell) and, with few warps on the SM, the latency
// of the exchange; loading and storing cost 0.03 us per KB of the tiles on an
// SM, hidden behind other tiles where the SM holds more than one.
inline double tile_us(const TileShape& t, int T, const BlockGrids& g, int sms,
                      const TileCost& c = TileCost{})
{
    const int vw = tile_vw(t, T), vh = tile_vh(t, T);
    if (vw < 8 || vh < 2) return 0.0;
    const double n = (double)((g.blocks(vw, vh) + sms - 1) / sms);  // tiles of the busiest SM
    const int occ = t.maxw / t.nw;
    const double k = std::min(n, (double)occ), rounds = std::max(1.0, n / occ);
    const double level = 4.0 * t.nw * t.R * t.C / 1965.0 * 1.04 * c.level * (t.C == 2 && t.R == 8 ? c.two : 1.0) *
                         (t.R == 4 ? c.four : 1.0) *
                         (t.maxw <= 12 ? 0.95 : 1.0);  // (registers to overlap rows)
    const double kb = k * t.nw * t.R * t.C * 32 * 8 / 1024.0 * 0.03 * c.bytes;
    const double lat = (k * t.nw <= 12 ? 0.08 : 0.03) * c.latency;
    return 1.0 + n * T * level + (occ == 1 ? rounds : 1.0) * kb + (n - k) * 0.4 + lat * T * rounds;
}

// Rows of a stream's strip: the fewest that fill no more than one wave of
// eight warps per SM (the whole grid's where even those make more strips).
inline int stream_rows(const BlockGrids& g, int sms)
{
    int lo = 1, hi = g.rows();
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (g.blocks(kStreamW, mid) <= 8LL * sms) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// The cheapest tile for one launch of T levels.
template <int NSHAPE>
inline TileShape best_tile(const TileShape (&shapes)[NSHAPE], int T, const BlockGrids& g, int sms,
                           double* us, const TileCost& cost = TileCost{})
{
    TileShape best = shapes[0];
    *us = 1e300;
    for (const TileShape& t : shapes) {
        const double one = tile_us(t, T, g, sms, cost);
        if (one > 0 && one < *us) {
            *us = one;
            best = t;
        }
    }
    return best;
}

// The cheapest way to run nlevels levels in tiles.
template <int NSHAPE>
inline BlockPlan plan_tiles(const TileShape (&shapes)[NSHAPE], const BlockGrids& g, int nlevels,
                            int step, int maxT, int sms, const TileCost& cost = TileCost{})
{
    BlockPlan best{false, step, 1e300};
    for (int T = step; T <= std::min(maxT, kTileMaxT); T += step) {
        const int k = (nlevels + T - 1) / T;
        const int Tk = ((nlevels + k - 1) / k + step - 1) / step * step;  // even shares
        double one;
        best_tile(shapes, Tk, g, sms, &one, cost);
        if (k * one < best.us) best = BlockPlan{false, Tk, k * one};
    }
    return best;
}

// The cheapest way to run nlevels levels.  Streams win from about 2000² up
// (us per level in runs of 480, stream / best tile: 1120² 2.08 / 1.33, 2048² 4.02 /
// 4.05, 4096² 11.6 / 15.7, 8192² 42.4 / 60.0); below, the tile whose count fits the
// SMs best.
template <int NSHAPE>
inline BlockPlan plan_block(const TileShape (&shapes)[NSHAPE], const BlockGrids& g, int nlevels,
                            int step, int maxT, int sms, const TileCost& cost = TileCost{})
{
    BlockPlan best = plan_tiles(shapes, g, nlevels, step, maxT, sms, cost);
    if (nlevels >= kStreamT && maxT >= kStreamT) {
        const int rows = stream_rows(g, sms);
        // (strips of very wide grids, or of many, may fill more than one wave)
        const double waves = std::max(1.0, (double)g.blocks(kStreamW, rows) / (8.0 * sms));
        double us = nlevels / kStreamT * (10.2 + 0.645 * rows) * waves * cost.stream, tail = 0.0;
        const int rest = (nlevels % kStreamT + step - 1) / step * step;
        if (rest) best_tile(shapes, rest, g, sms, &tail, cost);
        if (us + tail < best.us) best = BlockPlan{true, kStreamT, us + tail};
    }
    return best;
}

// Levels of the next launch with `left` levels to go: streams while there are
// enough, tiles in even shares.
inline int plan_next(const BlockPlan& p, long long left, int step)
{
    if (p.stream) return left >= kStreamT ? kStreamT : (int)((left + step - 1) / step * step);
    const long long k = (left + p.T - 1) / p.T;
    return (int)(((left + k - 1) / k + step - 1) / step * step);
}

// --------------------------------------------------------------- launches --
template <class S, bool RK2, int C, int R, int MAXW>
inline void launch_tile(const BlockArgs& a, int nw, cudaStream_t st)
{
    auto k = heat_block_tile<S, RK2, C, R, MAXW>;
    const size_t smem = tile_smem<C>(nw);
    if (smem > 48 * 1024) allow_big_smem(k);
    launch_after(k, a.units, 32 * nw, smem, st, a);
}

template <class S, bool RK2>
inline void launch_block_tile(const TileShape& t, BlockArgs a, int T, cudaStream_t st)
{
    a.T = T;
    a.vw = tile_vw(t, T);
    a.vh = tile_vh(t, T);
    a.ncs = (a.ny + a.vw - 1) / a.vw;
    a.units = a.ncs * ((a.nx + a.vh - 1) / a.vh);
    if constexpr (RK2) {
        if (t.C == 4 && t.R == 8) launch_tile<S, RK2, 4, 8, 12>(a, t.nw, st);
        else if (t.R == 6) launch_tile<S, RK2, 4, 6, 12>(a, t.nw, st);
        else if (t.C == 4) launch_tile<S, RK2, 4, 4, 16>(a, t.nw, st);
        else if (t.R == 8) launch_tile<S, RK2, 2, 8, 16>(a, t.nw, st);
        else launch_tile<S, RK2, 2, 4, 24>(a, t.nw, st);
    } else {
        if (t.R == 10) launch_tile<S, RK2, 4, 10, 12>(a, t.nw, st);
        else if (t.C == 4 && t.R == 8) launch_tile<S, RK2, 4, 8, 16>(a, t.nw, st);
        else if (t.C == 4) launch_tile<S, RK2, 4, 6, 16>(a, t.nw, st);
        else if (t.R == 8) launch_tile<S, RK2, 2, 8, 20>(a, t.nw, st);
        else launch_tile<S, RK2, 2, 4, 24>(a, t.nw, st);
    }
}

template <class S, bool RK2>
inline void launch_block_stream(BlockArgs a, int sms, cudaStream_t st)
{
    a.T = kStreamT;
    a.vw = kStreamW;
    a.ncs = (a.ny + a.vw - 1) / a.vw;
    const BlockGrid g{a.nx, a.ny};
    a.vh = stream_rows(BlockGrids{&g, 1}, sms);
    a.units = a.ncs * ((a.nx + a.vh - 1) / a.vh);
    launch_after(heat_block_stream<S, RK2>, a.units, 32, 0, st, a);
}

// ------------------------------------------------------------------ batch --
// Many grids in one launch: block g is unit units[g].y of grid units[g].x.
struct BlockInst {
    double* base[2];
    double cr;
    int nx, ny;
};

__device__ __forceinline__ void batch_block_args(const BlockInst* inst, int i, int par, int T,
                                                 int vw, int vh, BlockArgs& a)
{
    const BlockInst b = inst[i];
    a.in = b.base[par];
    a.out = b.base[1 - par];
    a.out1 = nullptr;
    a.nx = b.nx;
    a.ny = b.ny;
    a.T = T;
    a.vw = vw;
    a.vh = vh;
    a.ncs = (b.ny + vw - 1) / vw;
    a.units = 0;
    a.v4 = b.ny % 4 == 0;
    a.nframe = 0;
    a.cr = b.cr;
}

template <class S>
__global__ void __launch_bounds__(32, 8)
    heat_block_stream_batch(const BlockInst* __restrict__ inst, const int2* __restrict__ units,
                            int par, int vh)
{
    __shared__ __align__(16) S ring[kBlockRing * 32 * kStreamC];
    const int2 u = units[blockIdx.x];
    BlockArgs a;
    batch_block_args(inst, u.x, par, kStreamT, kStreamW, vh, a);
    grid_wait();
    grid_release();
    block_stream_body<S, false>(a, u.y, ring);
}

template <int C, int R, int MAXW>
__global__ void __launch_bounds__(32 * MAXW, 1)
    heat_block_tile_batch(const BlockInst* __restrict__ inst, const int2* __restrict__ units,
                          int par, int T, int vw, int vh)
{
    extern __shared__ __align__(16) double tile_sm[];
    const int2 u = units[blockIdx.x];
    BlockArgs a;
    batch_block_args(inst, u.x, par, T, vw, vh, a);
    grid_wait();
    block_tile_body<double, false, C, R>(a, u.y, blockDim.x >> 5, tile_sm);
}

}  // namespace psb
