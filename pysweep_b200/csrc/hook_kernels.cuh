// Kernels around a user step hook, compiled at run time (NVRTC, sm_100a) with
// the hook's source.  Host side: hook.cuh.
//
// The reference includes the plugin's
//     __device__ void step(double* shared_state, int idx, int globalTimeStep)
// textually into its phase kernels (pysweep/core/pysweep.cu:25,
// pysweep/core/io.py:146-155) and gives it the framework constants VARS,
// TIMES, MPSS, MOSS, NV, OPS, ITS, SX, SY as __constant__ ints
// (pysweep/core/pysweep.cu:12-20): the hook reads variable v of the cell at
// idx + v*VARS, its neighbours at idx +- SY (rows) and idx +- 1 (columns),
// the previous level at idx - TIMES and writes the next one at idx + TIMES.
//
// Here the hook runs inside the same swept phases as the built-in equations
// (stream_body and seam_body of swept.cuh, with the LINEAR slot layout that
// keeps the previous, current and next level at one stride) and inside
// overlapped blocks.  Each kernel kind has its own tile geometry, so the
// generated source includes the hook once per kind, in the namespaces
// psh_stream, psh_seam and psh_std, each with its own framework constants
// (set by the host before every run) and its own copy of the hook's
// __constant__ globals (set together by name).  The prelude defines
// PSH_OPS, PSH_ITS, PSH_NV and the block tiles (PSH_BLK_W columns at level 1,
// PSH_BLK_NT threads, at most PSH_BLK_MAXT levels) before including this file.
#pragma once
#include "swept.cuh"

namespace psb {

// The hook as a built-in equation functor: u points at the cell of the
// current level; the next and previous levels sit TIMES elements after and
// before it in the tile (the namespace's layout guarantees this), so u is
// passed as the shared array with idx = 0.
struct HookStream {
    static constexpr int OPS = PSH_OPS;
    __device__ static __forceinline__ void step(const double* u, const double*, double*, const Nbr&,
                                                int gts, int, const EqParams&)
    {
        psh_stream::step(const_cast<double*>(u), 0, gts);
    }
};

struct HookSeam {
    static constexpr int OPS = PSH_OPS;
    __device__ static __forceinline__ void step(const double* u, const double*, double*, const Nbr&,
                                                int gts, int, const EqParams&)
    {
        psh_seam::step(const_cast<double*>(u), 0, gts);
    }
};

// Block tiles (psh_block): SX x SY cells per variable with kBlkCols columns,
// slots of levels -1, 0, 1, .. one after another: TIMES = one slot, VARS = one
// variable plane, SY = one tile row.
constexpr int kBlkCols = PSH_BLK_W + 2 * PSH_OPS, kBlkNT = PSH_BLK_NT;

}  // namespace psb

using psb::SweptArgs;

// The streams (UpPyramid / XBridge), TIMES = slot + OPS: level m's column k
// sits OPS columns right of level m-1's (the chunk's parallelogram).
#define PSH_STREAM(NAME, W, GAP)                                                                  \
    extern "C" __global__ void __launch_bounds__(256) NAME(SweptArgs a)                         \
    {                                                                                             \
        extern __shared__ double psh_sm[];                                                        \
        psb::stream_body<psb::HookStream, PSH_ITS, W, GAP, 256, true>(a, blockIdx.x, psh_sm);    \
    }
PSH_STREAM(psh_prism32, 32, false)
PSH_STREAM(psh_gap32, 32, true)
PSH_STREAM(psh_prism64, 64, false)
PSH_STREAM(psh_gap64, 64, true)
#undef PSH_STREAM

// The seams (YBridge / Octahedron), TIMES = one slot.
extern "C" __global__ void __launch_bounds__(128) psh_ybridge(SweptArgs a)
{
    extern __shared__ double psh_sm[];
    psb::seam_body<psb::HookSeam, PSH_ITS, false, 128, double, true>(a, blockIdx.x, psh_sm);
}

extern "C" __global__ void __launch_bounds__(128) psh_octahedron(SweptArgs a)
{
    extern __shared__ double psh_sm[];
    psb::seam_body<psb::HookSeam, PSH_ITS, true, 128, double, true>(a, blockIdx.x, psh_sm);
}

// T levels of an overlapped block (T = 1: one level of the standard
// decomposition, pysweep/core/pysweep.cu:259-275).  The tile's newest level (and
// the one before it, where `older` is given) with a periodic halo of OPS cells
// per level into shared memory, two columns per load where rows and addresses
// allow; level m on the rows and columns that are still exact, a warp to a row;
// the last level's exact cells back (two base levels: the one before it, too),
// and every level that a frame keeps.  Level 1 spans PSH_BLK_W columns, so that
// no warp's pass over a row runs nearly empty.
// What bounds it: the hook's shared-memory reads (heat: five reads and a write
// for eight FP64 operations), and the tile's way in and out: a hook that only
// copies takes three quarters of heat's time.  Heat as a hook, 200 levels at
// 1024²: prisms of blocksize 16 3.67 ms, here 0.85; with one column per load and
// a division per row and variable 0.97.
struct HookFrames {
    double* level[PSH_BLK_MAXT];
};

extern "C" __global__ void __launch_bounds__(psb::kBlkNT)
    psh_block(const double* newest, const double* older, double* out, double* out1,
              HookFrames frames, int any_frame, int nx, int ny, int T, int rows1, int gts)
{
    using namespace psb;
    constexpr int OPS = PSH_OPS, NV = PSH_NV, CC = kBlkCols;
    extern __shared__ __align__(16) double t[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, NW = blockDim.x >> 5;
    const int RR = rows1 + 2 * OPS, SL = NV * RR * CC;  // tile rows, one slot
    const int ih = rows1 - 2 * OPS * (T - 1), iw = PSH_BLK_W - 2 * OPS * (T - 1);
    const int x0 = blockIdx.y * ih, y0 = blockIdx.x * iw;
    const size_t vs = (size_t)nx * ny;
    // two columns at once: tile and grid columns of one parity and rows of whole
    // pairs (y0, CC and iw are even; a state is 16-byte aligned where its user's
    // buffer is)
    const bool pairs = ny % 2 == 0 && OPS * T % 2 == 0 &&
                       (((size_t)newest | (size_t)older | (size_t)out | (size_t)out1) & 15) == 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto load = [&](int i, int k, bool two) {  // tile row i, column k (and the next)
        const size_t o = (size_t)wrap(x0 - OPS * T + i, nx) * ny + wrap(y0 - OPS * T + k, ny);
        double* to = t + SL + i * CC + k;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            double* q = to + v * RR * CC;
            if (two) {
                cp_async16(q, newest + v * vs + o);
                if (older) cp_async16(q - SL, older + v * vs + o);
            } else {
                cp_async8(q, newest + v * vs + o);
                if (older) cp_async8(q - SL, older + v * vs + o);
            }
        }
    };
    if (pairs)
        for (int e = threadIdx.x; e < RR * (CC / 2); e += blockDim.x)
            load(e / (CC / 2), e % (CC / 2) * 2, true);
    else
        for (int e = threadIdx.x; e < RR * CC; e += blockDim.x) load(e / CC, e % CC, false);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    // the exact cells of level m to global memory
    auto store = [&](double* dst, int m, bool two) {
        const double* src = t + (m + 1) * SL + OPS * T * (CC + 1);
        const int rows = min(ih, nx - x0), cols = min(iw, ny - y0);
#pragma unroll
        for (int v = 0; v < NV; ++v)
            for (int i = w; i < rows; i += NW) {
                double* row = dst + v * vs + (size_t)(x0 + i) * ny + y0;
                const double* from = src + (v * RR + i) * CC;
                if (two) {
                    for (int k = 2 * lane; k < cols; k += 64)
                        *reinterpret_cast<double2*>(row + k) = *reinterpret_cast<const double2*>(from + k);
                } else {
                    for (int k = lane; k < cols; k += 32) row[k] = from[k];
                }
            }
    };
    for (int m = 1; m <= T; ++m) {
        const int lo = OPS * m;
        for (int i = lo + w; i < RR - lo; i += NW)
            for (int k = lo + lane; k < CC - lo; k += 32) psh_std::step(t, m * SL + i * CC + k, gts + m - 1);
        __syncthreads();
        if (any_frame && frames.level[m - 1]) store(frames.level[m - 1], m, false);
    }
    store(out, T, pairs);
    if (out1) store(out1, T - 1, pairs);
}
