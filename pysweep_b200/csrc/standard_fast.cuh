// Standard decomposition for the heat equation (one variable): one level per
// launch (pysweep/core/pysweep.cu:259-275 computes the same step with one thread
// per cell and padded halos).
//
// A warp owns a 64-column strip of RB rows; lane l holds columns 2l, 2l+1.  It
// loads its rows, the one above and the one below at once, so a launch waits for
// memory once, and takes the left / right neighbours from the adjacent lanes by
// shuffle (lanes 0 and 31 load theirs).  Arithmetic: Heat in equations.cuh.
// Bound by HBM where the fields exceed L2 (16 bytes per cell: 428 G cells/s at
// 8192² in a short run, 106% of the measured copy's rate, the halo rows coming from
// L2; 405 in one of 5000 levels), below
// by the launch and one round trip.  us per level, against rows streamed one by
// one down 32-row strips: 2048² 14.4 -> 7.2, 4096² 49 -> 41, 8192² 182 -> 157;
// against one thread per cell (1120 columns are no multiple of 64): 7.4 -> 3.3.
// T is the storage type (double, or float with every level evaluated in
// double and rounded to float, as the reference's float32 runs do).
#pragma once
#include "heat_block.cuh"

namespace psb {

constexpr int kStdWarps = 4;

// Rows per warp: eight; four where eight leave the SMs fewer than 28 warps each
// (1120²: 3.5 against 3.8 us; 2048²: 7.75 against 7.4; before the warps were stacked).
inline int standard_rows(int nx, int ny, int sms)
{
    return (long long)((ny + 63) / 64) * ((nx + 7) / 8) < 28LL * sms ? 4 : 8;
}

// Whether a CTA's warps lie below one another, so that the rows they share come
// from L1, or side by side (us, side by side / below: 1152² 3.7 / 3.5, float32 4.0 /
// 3.3, 2048² 7.5 / 7.3; where a field is far larger than L2 8192² 156 / 159; where a
// full stage reads a second field 2048² 10.7 / 11.9).
inline bool standard_below(bool rk2, int nx, int ny) { return !rk2 && (long long)nx * ny <= 1 << 24; }

// CTAs of a level in rows of `rows` per warp.
inline int standard_grid(int nx, int ny, int rows, bool below)
{
    const int ncs = (ny + 63) / 64, nr = (nx + rows - 1) / rows;
    return below ? ncs * ((nr + kStdWarps - 1) / kStdWarps) : (ncs * nr + kStdWarps - 1) / kStdWarps;
}

template <bool RK2, int RB, class T>
__global__ void __launch_bounds__(32 * kStdWarps) heat_standard(const T* cur, const T* prev,
                                                                T* out, T* frame, int nx, int ny,
                                                                int gts, double cr, int below)
{
    using P = typename Pair2<T>::type;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ncs = (ny + 63) / 64;
    const int unit = below ? blockIdx.x : blockIdx.x * kStdWarps + warp, row = unit / ncs;
    const int x0 = below ? (row * kStdWarps + warp) * RB : row * RB;
    if (x0 >= nx) return;  // whole warp
    const int c0 = (unit - row * ncs) * 64 + 2 * lane;
    // (the last strip may reach past the row: it wraps; what lies further than
    // one row on, nobody reads)
    auto in_row = [&](int c) { return c < ny ? c : (c < 2 * ny ? c - ny : 0); };
    const int g = in_row(c0);
    const int hcol = lane == 0 ? (c0 == 0 ? ny - 1 : in_row(c0 - 1)) : in_row(c0 + 2);
    const bool edge = lane == 0 || lane == 31;
    const bool full = (gts % 2 == 0);
    grid_wait();
    double2 v[RB + 2], b[RK2 ? RB : 1];
    double h[RB];
    int r = x0 == 0 ? nx - 1 : x0 - 1;
#pragma unroll
    for (int i = 0; i < RB + 2; ++i) {
        const size_t o = (size_t)r * ny;
        v[i] = widen(*reinterpret_cast<const P*>(cur + o + g));
        if (i > 0 && i <= RB) {
            h[i - 1] = edge ? (double)cur[o + hcol] : 0.0;
            if constexpr (RK2)
                if (full) b[i - 1] = widen(*reinterpret_cast<const P*>(prev + o + g));
        }
        r = r + 1 >= nx ? r + 1 - nx : r + 1;
    }
    grid_release();
#pragma unroll
    for (int i = 0; i < RB; ++i) {
        const double2 up = v[i], ce = v[i + 1], dn = v[i + 2];
        double left = __shfl_up_sync(0xffffffffu, ce.y, 1);
        double right = __shfl_down_sync(0xffffffffu, ce.x, 1);
        if (lane == 0) left = h[i];
        if (lane == 31) right = h[i];
        double n0, n1;
        if (!RK2) {
            n0 = to_level<T>(heat_fe(ce.x, up.x, dn.x, left, ce.y, cr));
            n1 = to_level<T>(heat_fe(ce.y, up.y, dn.y, ce.x, right, cr));
        } else {
            // heat.py:53-57: coeff*cd + base, base = u[t-1] on full steps
            const double cd0 = __dadd_rn(__dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, ce.x, dn.x), up.x)),
                                         __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, ce.x, ce.y), left)));
            const double cd1 = __dadd_rn(__dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, ce.y, dn.y), up.y)),
                                         __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, ce.y, right), ce.x)));
            const double cf = full ? 1.0 : 0.5;
            n0 = to_level<T>(__dadd_rn(__dmul_rn(cf, cd0), full ? b[i].x : ce.x));
            n1 = to_level<T>(__dadd_rn(__dmul_rn(cf, cd1), full ? b[i].y : ce.y));
        }
        if (x0 + i < nx && c0 < ny) {
            const size_t o = (size_t)(x0 + i) * ny + c0;
            *reinterpret_cast<P*>(out + o) = pair2<T>(n0, n1);
            if (frame) *reinterpret_cast<P*>(frame + o) = pair2<T>(n0, n1);
        }
    }
}

}  // namespace psb
