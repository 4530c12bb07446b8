// Euler, one level per launch: warps march down strips of 64 columns.
//
// A warp holds two columns per lane and steps row by row, so a row's face is
// evaluated once and carried to the next row in registers, a column's face
// once by the lane on its left (the neighbour's share arrives by shuffle), and
// the rows wait in a ring in shared memory that cp.async fills ahead of them.
// 60 of the 64 columns are exact; a strip evaluates one row of faces more than
// it has rows.  No barrier, no face in shared memory.
//
// What bounds it: FP64 operations (537 per cell, of which 228 are fused
// multiply-adds that mostly read three register pairs, three cycles of the pipe
// each instead of two) and their latency of eight cycles; DRAM 64 to 96 bytes.
// A face needs 19 quotients and three square roots; the divisions were most of
// the instructions.  Seven quotients of a side share the denominator rho, two
// share sp0, so each denominator gets one reciprocal and every quotient four
// operations on it (quot); a cell's two limiter ratios are each other's inverse,
// and one of them needs no value but whether it exceeds 1e6 (limiters).  Every
// result is the correctly rounded one, so levels equal the per-cell step's
// (Euler::step) bitwise.  907 warp instructions per cell for the 1806 of tiles
// with their faces in shared memory; G cells/s, tiles / here: 480² 6.6 / 11.3,
// 1120² 8.8 / 18.5, 4096² 9.2 / 22.3.  Rows with a value outside the safe ranges
// below take plain divisions, as all do where a constant is: 480² 7.7, 1120² 10.4,
// 2048² 12.5 (called instead of inline 6.0, 8.3, 9.3).
#pragma once
#include <cmath>

#include "equations.cuh"
#include "heat_block.cuh"

namespace psb {
namespace euler {

// 1/b rounded correctly (y), and what is missing to 1/b (e).  From an
// approximation y0 good to 2^-20 (the rcp.approx.ftz.f64 instruction), with r = 1 -
// b y0: 1/b = y0/(1 - r), the geometric series y0 (1 + r + r^2 + ..) (M. J. Flynn,
// "On division by functional iteration", IEEE Trans. Computers C-19, 1970), here
// three terms of it by Horner's rule, good to 2^-60; then a step that rounds
// correctly (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  Take b in [1, 2), so ulps of 1/b are 2^-53, and D
// the distance of 1/b from the nearest midpoint of two doubles.  1 - b m is a
// nonzero multiple of 2^-106 for a midpoint m, so D is at least 2^-53/b ulps.  The
// series rounds a value within 2^-7 ulps of 1/b, so it is off by at most 1/2 + D
// ulps where D < 2^-7 (and by less than 0.51 elsewhere); the last step's value
// before rounding is then off by b (1/2 + D)^2 2^-53 ulps, less than D for every b
// but the largest, 2 - 2^-52, whose reciprocal may come out one ulp low: its last
// bit is set here.
struct Recip {
    double b, y, e;
};
__device__ __forceinline__ double recip_rn(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double r = __fma_rn(-b, y, 1.0), y1 = __fma_rn(y, r, y);
    y = __fma_rn(y1, r, y);
    y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
    const unsigned ones = ((unsigned)__double2hiint(b) | 0xfff00000u) & (unsigned)__double2loint(b);
    return __hiloint2double(__double2hiint(y), __double2loint(y) | (ones == 0xffffffffu ? 1 : 0));
}
__device__ __forceinline__ Recip recip(double b)
{
    Recip r;
    r.b = b;
    r.y = recip_rn(b);
    r.e = __dmul_rn(__fma_rn(-b, r.y, 1.0), r.y);
    return r;
}
// a/b rounded correctly: q0 = a y + a e rounds a value within 2^-51 ulp of a/b,
// so it is off by no more than 1/2 + D ulps (D as above, for a/b); its remainder
// a - b q0 is exact, and q0 + (a - b q0) y is off a/b by (1/2 + D) b |y - 1/b|
// ulps.  With y the rounded reciprocal that is less than D, which is at least
// 2^-53/b, for every b.  (A zero comes out as +0.)
__device__ __forceinline__ double quot(double a, const Recip& r)
{
    const double q0 = __fma_rn(a, r.y, __dmul_rn(a, r.e));
    return __fma_rn(__fma_rn(-r.b, q0, a), r.y, q0);
}
// N quotients by one denominator, each operation for all of them in turn: they
// share an operand, and a fused multiply-add that reads three register pairs
// takes three cycles of the pipe instead of two unless one of them is the
// previous one's (measured: 12.0 against 17.0 T/s).
template <int N>
__device__ __forceinline__ void quots(const double (&a)[N], const Recip& r, double (&q)[N])
{
    double m[N];
#pragma unroll
    for (int i = 0; i < N; ++i) m[i] = __dmul_rn(a[i], r.e);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = __fma_rn(a[i], r.y, m[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) m[i] = __fma_rn(-r.b, q[i], a[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = __fma_rn(m[i], r.y, q[i]);
}
// Ranges in which no step above or below over- or underflows.  A cell: rho in
// [2^-79, 2^79], the other variables zero or in [2^-115, 2^79]; a limiter factor
// zero or at least 2^-50.  A face's states then have rho in [2^-80, 2^80] and the
// rest zero (by cancellation, too: a sum of two doubles is zero or no smaller
// than their last place) or in [2^-170, 2^80], and the smallest numerator, a
// squared momentum of the Roe average, stays above 2^-930.  Rows with other
// cells take the plain divisions.  Words of |x|, so that zero is the largest:
__device__ __forceinline__ unsigned var_word(double x)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return (h | (unsigned)__double2loint(x)) ? h : 0x3ff00000u;  // (zero is in range)
}
__device__ __forceinline__ bool unsafe_rho(double x)
{
    return (unsigned)(__double2hiint(x) - 0x3b000000) >= 0x44e00000u - 0x3b000000u;
}
__device__ __forceinline__ bool unsafe_var(double x)
{
    return var_word(x) - 0x38c00000u >= 0x44e00000u - 0x38c00000u;
}
// The limiter factors min(Pr, 1)/2 (euler.py:250-256) of a cell between the
// pressure steps lo and up: hl for its upper face, Pr = up/lo; hr for its
// lower face, Pr = lo/up.  The ratio of the smaller to the larger step is
// divided out; the other is at least 1 wherever it is positive, so its factor
// is 1/2, or 0 above 1e6 (divided out only next to that line).  No step either
// way: 0/0, both factors 0.  Returns whether a factor is unsafe (see above).
__device__ __forceinline__ bool limiters(double lo, double up, double& hl, double& hr)
{
    const bool a = fabs(up) < fabs(lo);
    const double num = a ? up : lo, den = a ? lo : up;
    const double r = __ddiv_rn(num, den);
    double hb = r > 1.1e-6 ? 0.5 : 0.0;
    if (r > 0.9e-6 && r <= 1.1e-6) hb = __ddiv_rn(den, num) > 1e6 ? 0.0 : 0.5;
    const double hs = r >= 0.0 ? __dmul_rn(r, 0.5) : 0.0;  // (NaN: 0)
    hl = a ? hs : hb;
    hr = a ? hb : hs;
    return r > 0.0 && r < 0x1p-49;
}

// One side of a face: flux terms of the state Q in direction DIR and the
// quotients of its conserved variables by the density.
template <int DIR>
__device__ __forceinline__ void side(double gm1, const double* Q, double& p, double& nn, double& nt,
                                     double& ne, double* t)
{
    constexpr int A = DIR;
    const Recip r = recip(Q[0]);
    const double q11 = __dmul_rn(Q[1], Q[1]), q22 = __dmul_rn(Q[2], Q[2]);
    // s/(2 rho) = (s/rho)/2 exactly
    const double n[6] = {__dadd_rn(q11, q22), A == 1 ? q11 : q22, __dmul_rn(Q[1], Q[2]),
                         Q[1], Q[2], Q[3]};
    double q[6];
    quots(n, r, q);
    p = __dmul_rn(gm1, __fma_rn(-0.5, q[0], Q[3]));
    nn = q[1];
    nt = q[2];
    t[1] = q[3];
    t[2] = q[4];
    t[3] = q[5];
    ne = quot(__dmul_rn(__dadd_rn(Q[3], p), Q[A]), r);
}

// Two faces, each between cells a and b (q and the factor of the side towards
// the face): flux f and spectral term s, the values of flux and spectral in
// equations.cuh.  PLAIN: some state of the warp's is out of the safe range.
template <int DIR, bool PLAIN>
__device__ __forceinline__ void faces2(double gamma, double gm1,
                                       const double (&qa)[2][4], const double (&qb)[2][4],
                                       const double (&ha)[2], const double (&hb)[2],
                                       double (&f)[2][4], double (&s)[2][4])
{
    constexpr int A = DIR, B = 3 - DIR;
    double L[2][4], R[2][4];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const double d = __dsub_rn(qb[k][v], qa[k][v]);
            L[k][v] = __dadd_rn(qa[k][v], __dmul_rn(ha[k], d));
            R[k][v] = __dsub_rn(qb[k][v], __dmul_rn(hb[k], d));  // + hb (qa - qb)
        }
    if constexpr (PLAIN) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            flux<DIR>(gm1, L[k], R[k], f[k]);
            spectral<DIR>(gamma, gm1, L[k], R[k], s[k]);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        double vl[4], vr[4], pl, nl, tl, el, pr, nr, tr, er;
        side<DIR>(gm1, L[k], pl, nl, tl, el, vl);
        side<DIR>(gm1, R[k], pr, nr, tr, er, vr);
        f[k][0] = __dadd_rn(L[k][A], R[k][A]);
        f[k][A] = __dadd_rn(__dadd_rn(__dadd_rn(nl, pl), nr), pr);
        f[k][B] = __dadd_rn(tl, tr);
        f[k][3] = __dadd_rn(el, er);
        const double rl = __dsqrt_rn(L[k][0]), rr = __dsqrt_rn(R[k][0]);
        const double m = __dmul_rn(rl, rr);
        const double denom = recip_rn(__dadd_rn(rl, rr));
        double sp[4];
#pragma unroll
        for (int v = 1; v < 4; ++v)
            sp[v] = __dmul_rn(__dadd_rn(__dmul_rn(rl, vl[v]), __dmul_rn(rr, vr[v])), denom);
        const Recip rm = recip(m);
        const double m1 = __dmul_rn(m, sp[1]), m2 = __dmul_rn(m, sp[2]), m3 = __dmul_rn(m, sp[3]);
        const double p = __dmul_rn(
            gm1, __fma_rn(-0.5, quot(__dadd_rn(__dmul_rn(m1, m1), __dmul_rn(m2, m2)), rm), m3));
        double rad = __dadd_rn(__dsqrt_rn(quot(__dmul_rn(gamma, p), rm)), fabs(sp[DIR]));
        if (isnan(rad)) rad = 0.0;
#pragma unroll
        for (int v = 0; v < 4; ++v) s[k][v] = __dmul_rn(rad, __dsub_rn(L[k][v], R[k][v]));
    }
}

}  // namespace euler

constexpr int kMarchW = 60;     // exact columns of a strip
constexpr int kMarchRing = 4;   // rows in shared memory: three in use, one arriving
constexpr int kMarchWarps = 12; // warps per SM (168 registers; 8 or 16: 16.3, 18.9 against 18.7)

struct MarchArgs {
    const double* cur;
    const double* prev;
    double* out;
    double* frame;
    int nx, ny;
    int ncs, hs;  // column strips, rows of a strip
    int gts;
    double dtdx, dtdy, gamma, gm1;
};

// A warp's shared memory: rows of the strip, and what a row's face phase
// leaves for later: [0..3] its flux differences along x, [4..7] flux + spectral
// term of the face below the next row.
struct MarchShared {
    double ring[kMarchRing][4][64];
    double2 park[8][32];
};

// Strip `unit`: columns [cs kMarchW, +kMarchW), rows [rs hs, +hs).  PLAIN: every row
// takes the plain divisions (constants outside march_constants).
template <bool PLAIN>
__device__ __forceinline__ void march_body(const MarchArgs& a, int unit, MarchShared& sh)
{
    auto& ring = sh.ring;
    auto& park = sh.park;
    const int lane = threadIdx.x;
    const int nx = a.nx, ny = a.ny;
    const int cs = unit % a.ncs, rs = unit / a.ncs;
    const int x0 = rs * a.hs, x1 = min(x0 + a.hs, nx);
    const int clo = cs * kMarchW, chi = min(clo + kMarchW, ny);
    const int c0 = clo - 2 + 2 * lane;  // this lane's first column
    const int g = wrap(c0, ny);
    const size_t plane = (size_t)nx * ny;
    const double gamma = a.gamma, gm1 = a.gm1;
    const double hx = 0.5 * a.dtdx, hy = 0.5 * a.dtdy;
    const bool full = a.gts % 2 == 0;
    const bool mine = c0 >= clo && c0 < chi;
    const int n = x1 - x0 + 4;  // rows read: x0-2 .. x1+1
    int ir = wrap(x0 - 2, nx);
    grid_wait();
    auto issue = [&](int s) {
        if (s < n) {
            const double* src = a.cur + (size_t)ir * ny + g;
#pragma unroll
            for (int v = 0; v < 4; ++v) cp_async16(&ring[s % kMarchRing][v][2 * lane], src + v * plane);
            ir = ir + 1 == nx ? 0 : ir + 1;
        }
        cp_async_commit();
    };
    auto cells = [&](int s, double (&q)[2][4]) {  // the lane's cells of row s
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const double2 u = *reinterpret_cast<const double2*>(&ring[s % kMarchRing][v][2 * lane]);
            q[0][v] = u.x;
            q[1][v] = u.y;
        }
    };
    // pressures of row s; whether a cell of the warp's is out of the safe range
    auto pressures = [&](int s, double (&P)[2]) -> bool {
        double q[2][4];
        cells(s, q);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            bad |= euler::unsafe_rho(q[k][0]) | euler::unsafe_var(q[k][1]) |
                   euler::unsafe_var(q[k][2]) | euler::unsafe_var(q[k][3]);
        bad = __any_sync(0xffffffffu, bad);
#pragma unroll
        for (int k = 0; k < 2; ++k)
            P[k] = euler::pressure(gm1, q[k][0], q[k][1], q[k][2], q[k][3]);
        return bad;
    };
    auto limit2 = [&](const double (&lo)[2], const double (&up)[2], double (&hl)[2],
                      double (&hr)[2]) -> bool {
        const bool b0 = euler::limiters(lo[0], up[0], hl[0], hr[0]);
        const bool b1 = euler::limiters(lo[1], up[1], hl[1], hr[1]);
        return __any_sync(0xffffffffu, b0 | b1);
    };
#pragma unroll
    for (int s = 0; s < kMarchRing; ++s) issue(s);
    cp_async_wait<0>();  // rows x0-2 .. x0+1 are here
    __syncwarp();
    grid_release();
    // Pc, Pn: pressures of rows i and i+1; dn: the step between them; hl: the
    // factor of row i towards its upper face; badc, badn: unsafe rows; badl:
    // unsafe factors of row i
    double Pc[2], Pn[2], dn[2], hl[2];
    bool badc, badn, badl, below = false;  // below: `above` of the row before
    {
        double Pm[2], dm[2], unused[2];
        pressures(0, Pm);
        badc = pressures(1, Pc);
        badn = pressures(2, Pn);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            dm[k] = __dsub_rn(Pc[k], Pm[k]);
            dn[k] = __dsub_rn(Pn[k], Pc[k]);
        }
        badl = limit2(dm, dn, hl, unused);
#pragma unroll
        for (int v = 0; v < 4; ++v) park[4 + v][lane] = make_double2(0.0, 0.0);
    }
    // row i (ring row s) and the face above it
    for (int i = x0 - 1; i < x1; ++i) {
        const int s = i - x0 + 2;
        __syncwarp();
        issue(s + 3);  // into the slot of row i-1
        cp_async_wait<1>();  // row i+2 is here
        __syncwarp();
        const size_t go = (size_t)(i < 0 ? 0 : i) * ny + g;
        double2 pv[4];
        if (full && i >= x0 && mine) {
#pragma unroll
            for (int v = 0; v < 4; ++v) pv[v] = *reinterpret_cast<const double2*>(a.prev + v * plane + go);
        }
        double Pf[2], df[2], hn[2], hr[2];
        const bool badf = pressures(s + 2, Pf);
#pragma unroll
        for (int k = 0; k < 2; ++k) df[k] = __dsub_rn(Pf[k], Pn[k]);
        const bool badm = limit2(dn, df, hn, hr);
        const bool above = PLAIN || (badc | badn | badl | badm);  // plain divisions for the face above row i
        {
            double q[2][4], qn[2][4], f[2][4], t[2][4];
            cells(s, q);
            cells(s + 1, qn);
            if (above) euler::faces2<1, true>(gamma, gm1, q, qn, hl, hr, f, t);
            else euler::faces2<1, false>(gamma, gm1, q, qn, hl, hr, f, t);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double2 lo = park[4 + v][lane];
                double D[2], G[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    D[k] = __dsub_rn(__dsub_rn(k ? lo.y : lo.x, f[k][v]), t[k][v]);
                    G[k] = __dadd_rn(__dadd_rn(0.0, f[k][v]), t[k][v]);
                }
                park[v][lane] = make_double2(D[0], D[1]);
                park[4 + v][lane] = make_double2(G[0], G[1]);
            }
        }
        if (i >= x0) {
            // faces between columns: 0 between the lane's two, 1 towards the
            // next lane's first
            double lo[2], up[2], l[2], r[2];
            up[0] = lo[1] = __dsub_rn(Pc[1], Pc[0]);
            up[1] = __dsub_rn(__shfl_down_sync(0xffffffffu, Pc[0], 1), Pc[1]);
            lo[0] = __shfl_up_sync(0xffffffffu, up[1], 1);
            const bool plain = limit2(lo, up, l, r) | badc | above | below;
            const double h[2] = {r[1], __shfl_down_sync(0xffffffffu, r[0], 1)};
            double q[2][4], qn[2][4], o[2][4];
            cells(s, q);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                qn[0][v] = q[1][v];
                qn[1][v] = ring[s % kMarchRing][v][min(2 * lane + 2, 63)];
            }
            // The stage: u + d/2 or the level before + d, d = (dx/2) dt/dx + (dy/2)
            // dt/dy of the flux differences dx, dy.  Of states in the safe ranges no
            // difference and no d is subnormal, so halving them is exact: it goes into
            // dt/dx and into a fused multiply-add.  (us per level at 1120²: so in every
            // row, which is wrong, 67.2; an arm for the other rows 67.8; a branch of
            // their own behind the faces 68.3.)
            auto row = [&](auto slow) {
                constexpr bool SLOW = decltype(slow)::value;
                double f[2][4], t[2][4];
                euler::faces2<2, SLOW>(gamma, gm1, q, qn, l, h, f, t);
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const double gi = __dadd_rn(__dadd_rn(0.0, f[0][v]), t[0][v]);
                    const double gl =
                        __shfl_up_sync(0xffffffffu, __dadd_rn(__dadd_rn(0.0, f[1][v]), t[1][v]), 1);
                    const double2 D = park[v][lane];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const double x = k ? D.y : D.x, y = __dsub_rn(__dsub_rn(k ? gi : gl, f[k][v]), t[k][v]);
                        const double d = SLOW ? __dadd_rn(__dmul_rn(__dmul_rn(x, 0.5), a.dtdx),
                                                          __dmul_rn(__dmul_rn(y, 0.5), a.dtdy))
                                              : __dadd_rn(__dmul_rn(x, hx), __dmul_rn(y, hy));
                        if (full) o[k][v] = __dadd_rn(k ? pv[v].y : pv[v].x, d);
                        else o[k][v] = SLOW ? __dadd_rn(q[k][v], __dmul_rn(0.5, d)) : __fma_rn(0.5, d, q[k][v]);
                    }
                }
            };
            if (PLAIN || plain) row(std::true_type());
            else row(std::false_type());
            if (mine) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    *reinterpret_cast<double2*>(a.out + v * plane + go) = make_double2(o[0][v], o[1][v]);
                    if (a.frame)
                        *reinterpret_cast<double2*>(a.frame + v * plane + go) =
                            make_double2(o[0][v], o[1][v]);
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            Pc[k] = Pn[k];
            Pn[k] = Pf[k];
            dn[k] = df[k];
            hl[k] = hn[k];
        }
        badc = badn;
        badn = badf;
        badl = badm;
        below = above;
    }
}

template <bool PLAIN>
__global__ void __launch_bounds__(32, kMarchWarps) euler_march(const __grid_constant__ MarchArgs a)
{
    __shared__ __align__(16) MarchShared sh;
    march_body<PLAIN>(a, blockIdx.x, sh);
}

// Many instances in one launch: block g is unit units[g].y of instance
// units[g].x.  slot: the level's place in an instance's base buffers, [base][2]
// fields; an instance counts its own levels.
struct MarchInst {
    double* base[2];
    double dtdx, dtdy, gamma, gm1;
    int nx, ny, level;
};

template <bool PLAIN>
__global__ void __launch_bounds__(32, kMarchWarps)
    euler_march_batch(const MarchInst* __restrict__ inst, const int2* __restrict__ units, int cur,
                      int prev, int out, int hs, int L)
{
    __shared__ __align__(16) MarchShared sh;
    const int2 u = units[blockIdx.x];
    const MarchInst b = inst[u.x];
    const size_t fe = (size_t)4 * b.nx * b.ny;
    MarchArgs a;
    a.cur = b.base[cur / 2] + cur % 2 * fe;
    a.prev = b.base[prev / 2] + prev % 2 * fe;
    a.out = b.base[out / 2] + out % 2 * fe;
    a.frame = nullptr;
    a.nx = b.nx;
    a.ny = b.ny;
    a.ncs = (b.ny + kMarchW - 1) / kMarchW;
    a.hs = hs;
    a.gts = b.level + L;
    a.dtdx = b.dtdx;
    a.dtdy = b.dtdy;
    a.gamma = b.gamma;
    a.gm1 = b.gm1;
    march_body<PLAIN>(a, u.y, sh);
}

// Rows of a strip: the fewest that fit one wave of warps, or 6 to 24 in several
// waves where those cost less.  A strip costs its rows and 0.6 more (a grid's
// last strips have what rows are left); of w waves, those after the first cost
// 0.92 each (strips that start one after the other read the field in order:
// 4096², G cells/s with strips of 164 rows 18.5, 48 20.8, 20 21.4, 6 20.0), and
// the last 0.55 more the emptier it is (1600², w = 1.02 15.4, w = 1 18.5).  Over
// grids of 480² to 4096² within 4% of the best strip.
inline int march_rows(const BlockGrids& g, int sms)
{
    constexpr double start = 0.6, later = 0.92, drain = 0.55;
    const double wave = (double)kMarchWarps * sms;
    auto cost = [&](int hs) {
        double w = 0.0;
        for (int i = 0; i < g.n; ++i) {
            const int rest = g.g[i].nx % hs;
            w += ((g.g[i].ny + kMarchW - 1) / kMarchW) *
                 (g.g[i].nx / hs + (rest ? (rest + start) / (hs + start) : 0.0)) / wave;
        }
        const double full = std::floor(w);
        const double tail = w > full && full >= 1.0 ? drain * (1.0 - (w - full)) / full : 0.0;
        return (hs + start) * (1.0 + later * std::max(0.0, w - 1.0) + tail);
    };
    int lo = 1, hi = g.rows();
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if ((double)g.blocks(kMarchW, mid) <= wave) hi = mid;
        else lo = mid + 1;
    }
    int best = lo;
    // (a count of strips that no height brings into one wave costs its waves)
    double least = g.blocks(kMarchW, lo) <= wave ? lo + start : cost(lo);
    for (int hs = 6; hs <= std::min(24, lo - 1); ++hs)
        if (cost(hs) < least) {
            least = cost(hs);
            best = hs;
        }
    return best;
}

// The constants for which the safe ranges above hold; with others every row takes
// the plain divisions.
inline bool march_constants(const EqParams& p)
{
    auto mid = [](double x) { return x >= 0x1p-20 && x <= 0x1p20; };
    auto step = [](double x) { return x == 0.0 || (x >= 0x1p-200 && x <= 0x1p200) || (x <= -0x1p-200 && x >= -0x1p200); };
    return mid(p.d[2]) && mid(p.d[3]) && step(p.d[0]) && step(p.d[1]);
}

}  // namespace psb
