// C ABI of the B200 swept space-time solver (declarations: include/pysweep_b200.h).
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdarg>
#include <functional>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/pysweep_b200.h"
#include "equations.cuh"
#include "swept.cuh"
#include "heat_block.cuh"
#include "heatvar_block.cuh"
#include "launch.cuh"
#include "standard_fast.cuh"
#include "euler_march.cuh"
#include "batch.cuh"
#include "hook.cuh"

namespace psb {

// ---------------------------------------------------------- standard ------
// One level of the standard decomposition (pysweep/core/pysweep.cu:259-275,
// functions.py:126-146): every cell of level L+1 from levels L and L-1, with
// periodic neighbours taken directly instead of through padded halos.
template <class Eq>
__global__ void __launch_bounds__(256) standard_kernel(const double* __restrict__ cur,
                                                       const double* __restrict__ prev,
                                                       double* __restrict__ out,
                                                       double* __restrict__ frame, int nx, int ny,
                                                       int nv, int gts, EqParams p)
{
    const int y = blockIdx.x * blockDim.x + threadIdx.x;
    const int x = blockIdx.y;
    if (y >= ny) return;
    Nbr n;
    n.vs = nx * ny;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        int xx = x + k - 2, yy = y + k - 2;
        xx += xx < 0 ? nx : (xx >= nx ? -nx : 0);
        yy += yy < 0 ? ny : (yy >= ny ? -ny : 0);
        n.x[k] = (xx - x) * ny;
        n.y[k] = yy - y;
    }
    const size_t c = (size_t)x * ny + y;
    if constexpr (Coords<Eq>::value)
        Eq::step_at(cur + c, prev + c, out + c, n, gts, nv, p, x, y);
    else
        Eq::step(cur + c, prev + c, out + c, n, gts, nv, p);
    if (frame) {
        for (int v = 0; v < nv; ++v) frame[c + (size_t)v * n.vs] = out[c + (size_t)v * n.vs];
    }
}

}  // namespace psb

using namespace psb;

struct ps_solver {
    int device = 0;
    int eq = 0;
    int nv = 1, nx = 0, ny = 0, ops = 1, its = 1, bs = 0;
    int mpss = 0;
    int dtype = PS_DTYPE_F64;
    size_t esize = sizeof(double);  // bytes per element of every field and face buffer
    // tiling
    int H = 0, nseg = 1, chunk = 32, threads = 128;
    // heatvar / heatvar adjoint: courant numbers, the segment's recomputed
    // Laplacians (ps_set_field; device memory the caller owns)
    double* field[3] = {nullptr, nullptr, nullptr};
    bool nseg_auto = true;  // choose the segment count per run until configured
    bool h_set = false;     // levels per half-cycle configured
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    // the gap stream runs beside the y-bridge seam on a high-priority side
    // stream (forked from and joined back into `stream` with two events)
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    // named plugin constants
    std::map<std::string, double> globals;
    // device buffers
    double* base[2] = {nullptr, nullptr};  // [its][nv][nx][ny] each
    int cur = 0;                           // which base holds the current levels
    bool have_state = false;
    double* xface = nullptr;
    size_t xface_n = 0;
    double* yface = nullptr;
    size_t yface_n = 0;
    double* ring[3] = {nullptr, nullptr, nullptr};
    int64_t launches = 0;
    std::string err;
    // optional per-kernel device timing (ps_profile): events around every launch
    bool profile = false;
    std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> pending;
    std::vector<cudaEvent_t> event_pool;
    double prof_ms[8] = {0};
    int64_t prof_n[8] = {0};
    // algorithmic cell updates per kernel kind, accumulated with prof_ms
    double prof_cells[8] = {0};
    // user step hook compiled at run time (ps_create_hook); nullptr for the
    // built-in equations
    HookModule* hook = nullptr;
    std::string hook_src;    // the hook's source (declared types of its constants)
    std::string launch_err;  // a driver-API launch failure, reported by check_launch
};

namespace {

const char* kVersion = "pysweep_b200 0.1.0 (sm_100a)";
thread_local std::string g_create_error;  // message of the last failed ps_create

int fail(ps_solver* s, int code, const char* fmt, ...)
{
    if (s) {
        va_list ap, ap2;
        va_start(ap, fmt);
        va_copy(ap2, ap);
        const int n = vsnprintf(nullptr, 0, fmt, ap);
        va_end(ap);
        std::string buf(n > 0 ? (size_t)n : 0, '\0');
        if (n > 0) vsnprintf(&buf[0], (size_t)n + 1, fmt, ap2);
        va_end(ap2);
        s->err = buf;  // any length: hook compiler logs included
    }
    return code;
}

#define PS_CUDA(s, call)                                                                       \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess)                                                                 \
            return fail((s), e_ == cudaErrorMemoryAllocation ? PS_ERR_NOMEM : PS_ERR_CUDA,     \
                        "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

size_t field_elems(const ps_solver* s) { return (size_t)s->nv * s->nx * s->ny; }
// element offsets and sizes in the solver's storage type (double or float;
// device buffers are kept as double* and addressed in bytes)
double* at(const ps_solver* s, double* p, size_t elems)
{
    return reinterpret_cast<double*>(reinterpret_cast<char*>(p) + elems * s->esize);
}
size_t nbytes(const ps_solver* s, size_t elems) { return elems * s->esize; }

int eq_ops(int eq, int ops)
{
    switch (eq) {
    case PS_EQ_HEAT: return 1;
    case PS_EQ_HALF: return 1;
    case PS_EQ_HEATVAR: return 1;
    case PS_EQ_HEATVAR_ADJ: return 1;
    case PS_EQ_HEATVAR_ADJMU: return 1;
    case PS_EQ_EULER: return 2;
    default: return ops;  // example / checker take the configured ops
    }
}

// Equation constants, computed on the host the way each plugin's set_globals
// computes its CPU globals (heat.py:37, euler.py:23-24).
EqParams make_params_g(int eq, const std::map<std::string, double>& globals)
{
    EqParams p;
    memset(&p, 0, sizeof p);
    auto g = [&](const char* k, double d) {
        auto it = globals.find(k);
        return it == globals.end() ? d : it->second;
    };
    switch (eq) {
    case PS_EQ_HEAT: {
        const double alpha = g("ALPHA", 1.0), dt = g("DT", 0.0), dx = g("DX", 1.0);
        p.d[0] = alpha * dt / dx / dx;
        p.i[0] = g("SCHEME", 1.0) != 0.0;
        break;
    }
    case PS_EQ_EULER: {
        const double dt = g("DT", 0.0), dx = g("DX", 1.0), dy = g("DY", dx);
        const double gamma = g("GAMMA", 1.4);
        p.d[0] = g("DTDX", dt / dx);
        p.d[1] = g("DTDY", dt / dy);
        p.d[2] = gamma;
        p.d[3] = g("GAM_M1", gamma - 1.0);
        break;
    }
    case PS_EQ_EXAMPLE:
    case PS_EQ_CHECKER: p.i[0] = g("SCHEME", 1.0) != 0.0; break;
    default: break;
    }
    return p;
}

EqParams make_params(const ps_solver* s)
{
    EqParams p = make_params_g(s->eq, s->globals);
    if (s->eq == PS_EQ_HEATVAR || s->eq == PS_EQ_HEATVAR_ADJ || s->eq == PS_EQ_HEATVAR_ADJMU) {
        p.i[1] = s->nx;
        p.i[2] = s->ny;
        auto it = s->globals.find("LEN");
        p.i[3] = it == s->globals.end() ? 0 : (int)it->second;
        p.f[0] = s->field[0];
        p.f[1] = s->field[1];
        p.f[2] = s->field[2];
        p.fs = (long long)s->nx * s->ny;
    }
    return p;
}

// Equation id of solvers running a user step hook (internal: ps_create_hook)
constexpr int PS_EQ_HOOK = 5;

// ------------------------------------------------------------ dispatch ----
using SweptLaunch = std::function<void(const SweptArgs&, int grid, size_t smem, cudaStream_t)>;
using StdLaunch = void (*)(const double*, const double*, double*, double*, int, int, int, int,
                           const EqParams&, cudaStream_t);

template <class Eq, int ITS, int W, bool GAP>
void launch_stream(const SweptArgs& a, int grid, size_t smem, cudaStream_t st)
{
    auto k = stream_kernel<Eq, ITS, W, GAP, 256>;
    allow_big_smem(k);
    k<<<grid, 256, smem, st>>>(a);
}

template <class Eq, int ITS, bool GAP>
void launch_seam(const SweptArgs& a, int grid, size_t smem, cudaStream_t st)
{
    // one-variable stencils: 64 threads per seam (the seams are issue-bound
    // on per-level loop work that every warp repeats; measured 1-2% faster
    // in total than 128); Euler keeps 128 for its four-variable tiles
    constexpr int NT = Eq::OPS == 1 ? 64 : 128;
    auto k = seam_kernel<Eq, ITS, GAP, NT>;
    allow_big_smem(k);
    k<<<grid, NT, smem, st>>>(a);
}

template <class Eq>
void launch_standard(const double* cur, const double* prev, double* out, double* frame, int nx,
                     int ny, int nv, int gts, const EqParams& p, cudaStream_t st)
{
    dim3 grid((ny + 255) / 256, nx);
    standard_kernel<Eq><<<grid, 256, 0, st>>>(cur, prev, out, frame, nx, ny, nv, gts, p);
}

struct SweptSet {
    SweptLaunch P, Y, G, O;
};

template <class Eq, int ITS, int W>
SweptSet make_set()
{
    return SweptSet{launch_stream<Eq, ITS, W, false>, launch_seam<Eq, ITS, false>,
                    launch_stream<Eq, ITS, W, true>, launch_seam<Eq, ITS, true>};
}

// (equation, ops, its, chunk) -> kernels; nullptr members = not built.
bool pick_swept(int eq, int ops, int its, int chunk, SweptSet* out)
{
#define PS_SET(EQ, OP, IT, W, T) \
    if (eq == EQ && ops == OP && its == IT && chunk == W) { *out = make_set<T, IT, W>(); return true; }
    PS_SET(PS_EQ_HEAT, 1, 1, 32, Heat)
    PS_SET(PS_EQ_HEAT, 1, 2, 32, Heat)
    PS_SET(PS_EQ_HEAT, 1, 1, 64, Heat)
    PS_SET(PS_EQ_HEAT, 1, 2, 64, Heat)
    PS_SET(PS_EQ_EULER, 2, 2, 32, Euler)
    PS_SET(PS_EQ_EULER, 2, 2, 64, Euler)
    PS_SET(PS_EQ_HALF, 1, 1, 32, Half)
    PS_SET(PS_EQ_HALF, 1, 2, 32, Half)
    PS_SET(PS_EQ_EXAMPLE, 1, 1, 32, ExampleT<1>)
    PS_SET(PS_EQ_EXAMPLE, 1, 2, 32, ExampleT<1>)
    PS_SET(PS_EQ_EXAMPLE, 2, 1, 32, ExampleT<2>)
    PS_SET(PS_EQ_EXAMPLE, 2, 2, 32, ExampleT<2>)
    PS_SET(PS_EQ_CHECKER, 1, 1, 32, CheckerT<1>)
    PS_SET(PS_EQ_CHECKER, 1, 2, 32, CheckerT<1>)
    PS_SET(PS_EQ_CHECKER, 2, 1, 32, CheckerT<2>)
    PS_SET(PS_EQ_CHECKER, 2, 2, 32, CheckerT<2>)
    PS_SET(PS_EQ_HEATVAR, 1, 1, 32, HeatVar)
    PS_SET(PS_EQ_HEATVAR, 1, 1, 64, HeatVar)
    PS_SET(PS_EQ_HEATVAR_ADJ, 1, 1, 32, HeatVarAdj)
    PS_SET(PS_EQ_HEATVAR_ADJ, 1, 1, 64, HeatVarAdj)
    PS_SET(PS_EQ_HEATVAR_ADJMU, 1, 1, 32, HeatVarAdjMu)
    PS_SET(PS_EQ_HEATVAR_ADJMU, 1, 1, 64, HeatVarAdjMu)
#undef PS_SET
    return false;
}

StdLaunch pick_standard(int eq, int ops)
{
    switch (eq) {
    case PS_EQ_HEAT: return launch_standard<Heat>;
    case PS_EQ_EULER: return launch_standard<Euler>;
    case PS_EQ_HALF: return launch_standard<Half>;
    case PS_EQ_EXAMPLE: return ops == 2 ? launch_standard<ExampleT<2>> : launch_standard<ExampleT<1>>;
    case PS_EQ_CHECKER: return ops == 2 ? launch_standard<CheckerT<2>> : launch_standard<CheckerT<1>>;
    case PS_EQ_HEATVAR: return launch_standard<HeatVar>;
    case PS_EQ_HEATVAR_ADJ: return launch_standard<HeatVarAdj>;
    case PS_EQ_HEATVAR_ADJMU: return launch_standard<HeatVarAdjMu>;
    default: return nullptr;
    }
}

int check_launch(ps_solver* s)
{
    if (!s->launch_err.empty()) {
        const std::string m = s->launch_err;
        s->launch_err.clear();
        return fail(s, PS_ERR_CUDA, "kernel launch: %s", m.c_str());
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(s, PS_ERR_CUDA, "kernel launch: %s", cudaGetErrorString(e));
    s->launches++;
    return PS_OK;
}

cudaEvent_t take_event(ps_solver* s)
{
    if (!s->event_pool.empty()) {
        cudaEvent_t e = s->event_pool.back();
        s->event_pool.pop_back();
        return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
}

// Kernel kinds for ps_profile_read: 0 prism stream, 1 Y-bridge seam, 2 gap
// stream, 3 octahedron seam, 4 standard step, 5 overlapped block.
template <class F>
int timed_launch(ps_solver* s, int kind, double cells, F&& launch, cudaStream_t st = nullptr)
{
    cudaEvent_t a = nullptr, b = nullptr;
    if (!st) st = s->stream;
    if (s->profile) {
        a = take_event(s);
        b = take_event(s);
        cudaEventRecord(a, st);
    }
    launch();
    int rc = check_launch(s);
    if (s->profile) {
        cudaEventRecord(b, st);
        s->pending.push_back({kind, {a, b}});
        s->prof_cells[kind] += cells;
    }
    return rc;
}

int drain_profile(ps_solver* s)
{
    for (auto& p : s->pending) {
        float ms = 0.f;
        cudaError_t e = cudaEventElapsedTime(&ms, p.second.first, p.second.second);
        if (e != cudaSuccess) return fail(s, PS_ERR_CUDA, "event timing: %s", cudaGetErrorString(e));
        s->prof_ms[p.first] += ms;
        s->prof_n[p.first] += 1;
        s->event_pool.push_back(p.second.first);
        s->event_pool.push_back(p.second.second);
    }
    s->pending.clear();
    return PS_OK;
}

int ensure_swept_buffers(ps_solver* s)
{
    const int O2 = 2 * s->ops;
    const int nb = s->nx / s->bs;
    const int HF = std::max(s->H - 1, 0);
    const size_t xn = (size_t)nb * HF * 2 * s->nv * O2 * s->ny;
    // two y-face buffers: prism -> y-bridge, gap -> octahedron (the y-bridge
    // and the gap stream run at the same time)
    const size_t yn = 2 * (size_t)nb * s->nseg * 2 * HF * s->nv * s->bs * O2;
    if (xn > s->xface_n) {
        if (s->xface) cudaFree(s->xface);
        s->xface = nullptr;
        s->xface_n = 0;
        if (xn) PS_CUDA(s, cudaMalloc(&s->xface, nbytes(s, xn)));
        s->xface_n = xn;
    }
    if (yn > s->yface_n) {
        if (s->yface) cudaFree(s->yface);
        s->yface = nullptr;
        s->yface_n = 0;
        if (yn) PS_CUDA(s, cudaMalloc(&s->yface, nbytes(s, yn)));
        s->yface_n = yn;
    }
    return PS_OK;
}

// Levels per half-cycle until configured: MPSS, except heat with forward
// Euler at bs 32.  The prisms, the row slabs' halo exchange and the adjoint's
// checkpoint segments count in them; overlapped blocks take as many levels per
// launch as suit the grid.  12 of 15 is what heat's callers have always been
// told (ps_get_tiling): saved tilings and segment lengths stay valid.  Results
// do not depend on the choice.
int default_levels(int eq, int its, int bs, int mpss)
{
    if ((eq == PS_EQ_HEAT || eq == PS_EQ_HEATVAR || eq == PS_EQ_HEATVAR_ADJMU) && its == 1 && bs == 32)
        return std::min(mpss, 12);
    return mpss;
}

// tile slots of the stream and seam kernels: a ring of its+1 for the built-in
// equations, levels -1 .. Hmax for a step hook (slot_count in swept.cuh)
int tile_slots(const ps_solver* s) { return s->hook ? s->H + 2 : s->its + 1; }

size_t stream_smem(const ps_solver* s)
{
    const int O2 = 2 * s->ops, RS = s->chunk + O2;
    return s->esize * ((size_t)tile_slots(s) * s->nv * s->bs * RS +
                       (size_t)(s->H + 1) * s->nv * s->bs * O2);
}


bool solver_seam_direct(const ps_solver* s)
{
    return seam_direct(s->bs, s->ops, s->nv, s->its, s->H, s->esize, tile_slots(s));
}

size_t seam_smem(const ps_solver* s)
{
    const int ns = tile_slots(s);
    if (solver_seam_direct(s))
        return s->esize * (size_t)ns * s->nv * s->bs * (2 * s->ops * (s->H + 1));
    return s->esize * std::max(seam_smem_elems(false, s->bs, s->ops, s->nv, s->its, s->H, ns),
                               seam_smem_elems(true, s->bs, s->ops, s->nv, s->its, s->H, ns));
}

// ------------------------------------------------------------ step hooks ----
// Driver-API launch of a hook kernel; a failure is kept for check_launch.
void hook_launch(ps_solver* s, CUfunction f, int gx, int gy, int nt, size_t smem,
                 cudaStream_t st, void** args)
{
    CUresult r = drv().launchKernel(f, gx, gy, 1, nt, 1, 1, (unsigned)smem, (CUstream)st, args,
                                    nullptr);
    if (r != CUDA_SUCCESS) s->launch_err = cu_error(r);
}

SweptSet hook_set(ps_solver* s)
{
    const int w = s->chunk == 64 ? 1 : 0;
    HookModule* h = s->hook;
    auto mk = [s](CUfunction f, int nt) {
        return [s, f, nt](const SweptArgs& a, int grid, size_t smem, cudaStream_t st) {
            SweptArgs copy = a;
            void* args[] = {&copy};
            hook_launch(s, f, grid, 1, nt, smem, st, args);
        };
    };
    return SweptSet{mk(h->prism[w], 256), mk(h->ybridge, 128), mk(h->gap[w], 256),
                    mk(h->octahedron, 128)};
}

// The framework constants of one kernel kind's tile (pysweep/core/pysweep.cu:
// 12-20, set by io.copyConstants, io.py:169-184): a tile of `rows` x `cols`
// cells per variable, levels `times` elements apart.
int hook_frame(ps_solver* s, int ns, int rows, int cols, int times)
{
    HookModule* h = s->hook;
    const int vals[FW_COUNT] = {rows * cols, times, s->mpss, 2 * s->mpss, s->nv,
                                s->ops,      s->its, rows,   cols};
    for (int f = 0; f < FW_COUNT; ++f) {
        CUresult r = hook_set_fw(h, ns, f, vals[f], (CUstream)s->stream);
        if (r != CUDA_SUCCESS)
            return fail(s, PS_ERR_CUDA, "hook constant %s: %s", kHookFw[f], cu_error(r).c_str());
    }
    return PS_OK;
}

// ------------------------------------------------- overlapped heat blocks ----
bool aligned32(const void* p) { return reinterpret_cast<uintptr_t>(p) % 32 == 0; }

// Heat through overlapped space-time blocks (heat_block.cuh): forward Euler
// with its 1, or the two-stage scheme with its 2.  maxT: levels per launch at
// most.  Two-stage levels run in pairs from a half stage on; a level left over
// on either side (a run that begins with a full stage, an odd count) is one
// standard step.
template <class S, bool RK2>
int run_block(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
              int frame_every, int maxT)
{
    constexpr int step = RK2 ? 2 : 1;
    const size_t fe = field_elems(s);
    const int its = s->its;
    const int every = frame_every > 0 ? frame_every : 1;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const EqParams prm = make_params(s);
    auto frame_of = [&](int64_t L) -> double* {
        if (!frames || L % its || (L / its) % every) return nullptr;
        const int64_t slot = (L / its) / every - 1;
        return slot < frame_cap ? at(s, frames, (size_t)slot * fe) : nullptr;
    };
    auto newest = [&](int b) { return at(s, s->base[b], (size_t)(its - 1) * fe); };
    int rc;
    int64_t done = 0;
    auto single = [&]() -> int {  // one level of the two-stage scheme
        const int b = s->cur;
        double* fr = frame_of(done + 1);
        const int gts = gts0 + (int)done;
        if (int e = timed_launch(s, 4, (double)s->nx * s->ny, [&] {
                launch_standard<Heat>(newest(b), s->base[b], newest(1 - b), fr, s->nx, s->ny, 1, gts,
                                      prm, s->stream);
            }))
            return e;
        PS_CUDA(s, cudaMemcpyAsync(s->base[1 - b], newest(b), nbytes(s, fe),
                                   cudaMemcpyDeviceToDevice, s->stream));
        s->cur = 1 - b;
        ++done;
        return PS_OK;
    };
    if (RK2 && nlevels > 0 && gts0 % 2 == 0 && (rc = single())) return rc;
    const int64_t last = RK2 ? nlevels - (nlevels - done) % 2 : nlevels;
    const BlockGrid grid{s->nx, s->ny};
    const BlockGrids grids{&grid, 1};
    BlockPlan plan{};
    BlockArgs a;
    memset(&a, 0, sizeof a);
    a.nx = s->nx;
    a.ny = s->ny;
    a.v4 = s->ny % 4 == 0;
    a.cr = prm.d[0];
    if (done < last) {
        const int n = (int)std::min<int64_t>(last - done, 1 << 20);
        const TileCost cost = RK2 ? kCostRK2 : (sizeof(S) == 4 ? kCostF32 : TileCost{});
        if constexpr (RK2) plan = plan_block(kTilesRK2, grids, n, step, maxT, sms, cost);
        else plan = plan_block(kTilesFE, grids, n, step, maxT, sms, cost);
    }
    // frames are stored by the block that computes their level where 4-wide
    // stores may reach them; else the block ends at the level and it is copied
    const bool direct = aligned32(frames);
    while (done < last) {
        int T = plan_next(plan, last - done, step);
        a.nframe = 0;
        double* copy_to = nullptr;
        for (int m = 1; m <= T; ++m) {
            double* f = frame_of(done + m);
            a.frame[m - 1] = direct ? f : nullptr;
            if (f && direct) ++a.nframe;
            if (f && !direct) {
                copy_to = f;
                T = m;
            }
        }
        a.in = newest(s->cur);
        a.out = newest(1 - s->cur);
        // the level before the newest is part of the state after the run
        a.out1 = RK2 && done + T == nlevels ? s->base[1 - s->cur] : nullptr;
        // frames and the kept level are stored by the tiles only
        const bool tile = !plan.stream || T < kStreamT || a.nframe || a.out1;
        if ((rc = timed_launch(s, 5, (double)s->nx * s->ny * T, [&] {
                 if (tile) {
                     double us;
                     if constexpr (RK2)
                         launch_block_tile<S, RK2>(best_tile(kTilesRK2, T, grids, sms, &us, kCostRK2), a, T, s->stream);
                     else
                         launch_block_tile<S, RK2>(best_tile(kTilesFE, T, grids, sms, &us), a, T, s->stream);
                 } else {
                     launch_block_stream<S, RK2>(a, sms, s->stream);
                 }
             })))
            return rc;
        s->cur = 1 - s->cur;
        done += T;
        if (copy_to)
            PS_CUDA(s, cudaMemcpyAsync(copy_to, newest(s->cur), nbytes(s, fe),
                                       cudaMemcpyDeviceToDevice, s->stream));
    }
    if (done < nlevels && (rc = single())) return rc;
    return PS_OK;
}

// Some field of a per-cell-courant solver lies off a 16-byte boundary.
bool var_odd(const ps_solver* s)
{
    for (const double* f : s->field)
        if (reinterpret_cast<uintptr_t>(f) % 16) return true;
    return false;
}

// The per-cell-courant equations in overlapped tiles (heatvar_block.cuh).
// Level L of the run has globalTimeStep gts0 + L - 1; the forward stores its old
// level's Laplacian at index gts - 1 of field 1, the adjoint reads index LEN -
// gts (ps_run has checked that they lie in it).  A frame ends its launch and is
// copied from the state.
template <int ROLE>
int run_var(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
            int frame_every)
{
    const size_t fe = field_elems(s), plane = (size_t)s->nx * s->ny;
    const int every = frame_every > 0 ? frame_every : 1;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const EqParams prm = make_params(s);
    const BlockGrid grid{s->nx, s->ny};
    VarArgs a;
    memset(&a, 0, sizeof a);
    a.C = prm.f[0];
    a.nx = s->nx;
    a.ny = s->ny;
    a.step = ROLE >= VAR_LAMBDA ? -(long long)plane : (long long)plane;
    const bool odd = var_odd(s);
    BlockPlan plan{};
    if (nlevels > 0)
        plan = plan_var<ROLE>(BlockGrids{&grid, 1}, (int)std::min<int64_t>(nlevels, 1 << 20), sms);
    int rc;
    for (int64_t done = 0; done < nlevels;) {
        int T = plan_next(plan, nlevels - done, 1);
        double* fr = nullptr;
        for (int m = 1; frames && m <= T; ++m)
            if ((done + m) % every == 0 && (done + m) / every - 1 < frame_cap) {
                fr = at(s, frames, (size_t)((done + m) / every - 1) * fe);
                T = m;
            }
        const int64_t gts = gts0 + done;  // of the launch's first level
        a.in = s->base[s->cur];
        a.out = s->base[1 - s->cur];
        if (ROLE == VAR_RECOMPUTE) a.lap = prm.f[1] + (gts - 1) * plane;
        if (ROLE >= VAR_LAMBDA) a.lap = prm.f[1] + (prm.i[3] - gts) * (int64_t)plane;
        if (ROLE == VAR_MU) a.g = prm.f[2];
        if (ROLE == VAR_LAMBDA) {
            // the second variable, from one base to the other
            a.g = s->base[1 - s->cur] + plane;
            PS_CUDA(s, cudaMemcpyAsync(a.g, s->base[s->cur] + plane, plane * sizeof(double),
                                       cudaMemcpyDeviceToDevice, s->stream));
        }
        if ((rc = timed_launch(s, 5, (double)plane * T,
                               [&] {
                                   if (odd) launch_var<ROLE, true>(a, T, sms, s->stream);
                                   else launch_var<ROLE>(a, T, sms, s->stream);
                               })))
            return rc;
        s->cur = 1 - s->cur;
        done += T;
        if (fr)
            PS_CUDA(s, cudaMemcpyAsync(fr, s->base[s->cur], nbytes(s, fe), cudaMemcpyDeviceToDevice,
                                       s->stream));
    }
    return PS_OK;
}

// Level by level in the base buffers: they hold 2 its levels, and each new one
// goes to the oldest slot, so no field is copied but after an odd count of
// two-stage levels.  launch(cur, prev, out, frame, gts) queues one level; prev is
// the level before cur (two base levels).  A frame that 16-byte stores cannot
// reach is copied from its level.
template <class F>
int run_levels(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
               int frame_every, int kind, F&& launch)
{
    const size_t fe = field_elems(s);
    const int its = s->its, every = frame_every > 0 ? frame_every : 1;
    double* slot[4];  // [base][its: older, newer]
    for (int q = 0; q < 2 * its; ++q) slot[q] = at(s, s->base[q / its], (size_t)(q % its) * fe);
    int older = its * s->cur, newest = older + its - 1;  // slots of levels L-2 and L-1
    for (int64_t L = 1; L <= nlevels; ++L) {
        const int next = (newest + 1) % (2 * its);
        double* fr = nullptr;
        if (frames && L % its == 0 && (L / its) % every == 0) {
            const int64_t k = (L / its) / every - 1;
            if (k < frame_cap) fr = at(s, frames, (size_t)k * fe);
        }
        const bool direct = reinterpret_cast<uintptr_t>(fr) % 16 == 0;
        int rc = timed_launch(s, kind, (double)s->nx * s->ny, [&] {
            launch(slot[newest], slot[older], slot[next], direct ? fr : nullptr, gts0 + (int)(L - 1));
        });
        if (rc) return rc;
        if (fr && !direct)
            PS_CUDA(s, cudaMemcpyAsync(fr, slot[next], nbytes(s, fe), cudaMemcpyDeviceToDevice,
                                       s->stream));
        older = newest;
        newest = next;
    }
    s->cur = newest / its;
    if (its == 2 && newest % 2 == 0) {
        // an odd count: the newest level moves up beside the one before it
        PS_CUDA(s, cudaMemcpyAsync(slot[newest + 1], slot[newest], nbytes(s, fe),
                                   cudaMemcpyDeviceToDevice, s->stream));
        PS_CUDA(s, cudaMemcpyAsync(slot[newest], slot[older], nbytes(s, fe), cudaMemcpyDeviceToDevice,
                                   s->stream));
    }
    return PS_OK;
}

// Euler level by level (euler_march.cuh), for either decomposition: its levels
// are bound by arithmetic, not by memory, so a cell evaluated twice costs more
// than a level kept on chip saves (prisms of blocksize 16 at 4096²: 6.3 G cell
// stages/s, at 1120² 5.1; level by level 21.4 and 18.7).
int run_march(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
              int frame_every, int kind)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const EqParams prm = make_params(s);
    const BlockGrid grid{s->nx, s->ny};
    MarchArgs a;
    memset(&a, 0, sizeof a);
    a.nx = s->nx;
    a.ny = s->ny;
    a.ncs = (s->ny + kMarchW - 1) / kMarchW;
    a.hs = march_rows(BlockGrids{&grid, 1}, sms);
    a.dtdx = prm.d[0];
    a.dtdy = prm.d[1];
    a.gamma = prm.d[2];
    a.gm1 = prm.d[3];
    const auto kernel = march_constants(prm) ? euler_march<false> : euler_march<true>;
    const int units = a.ncs * ((s->nx + a.hs - 1) / a.hs);
    return run_levels(s, nlevels, gts0, frames, frame_cap, frame_every, kind,
                      [&](const double* cur, const double* prev, double* out, double* fr, int gts) {
                          a.cur = cur;
                          a.prev = prev;
                          a.out = out;
                          a.frame = fr;
                          a.gts = gts;
                          launch_after(kernel, units, 32, 0, s->stream, a);
                      });
}

struct HookFrames {  // psh_block's argument (hook_kernels.cuh)
    double* level[kHookBlkMaxT];
};

// Queue one psh_block launch of T levels (its launch may overlap the end of the
// one before it).
void hook_block_launch(ps_solver* s, const HookBlock& b, int T, const double* newest,
                       const double* older, double* out, double* out1, HookFrames fr, int any_frame,
                       int gts)
{
    int nx = s->nx, ny = s->ny, rows = b.rows;
    const int ih = rows - 2 * s->ops * (T - 1), iw = kHookBlkW - 2 * s->ops * (T - 1);
    void* args[] = {&newest, &older, &out, &out1, &fr, &any_frame, &nx, &ny, &T, &rows, &gts};
    CUlaunchConfig cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDimX = (ny + iw - 1) / iw;
    cfg.gridDimY = (nx + ih - 1) / ih;
    cfg.gridDimZ = 1;
    cfg.blockDimX = T > 1 ? kHookBlkNT : b.threads1;
    cfg.blockDimY = cfg.blockDimZ = 1;
    cfg.sharedMemBytes = (unsigned)hook_block_smem(s->nv, s->ops, rows, T);
    cfg.hStream = (CUstream)s->stream;
    CUlaunchAttribute at;
    memset(&at, 0, sizeof at);
    at.id = CU_LAUNCH_ATTRIBUTE_PROGRAMMATIC_STREAM_SERIALIZATION;
    at.value.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    CUresult r = drv().launchKernelEx(&cfg, s->hook->block, args, nullptr);
    if (r != CUDA_SUCCESS) s->launch_err = cu_error(r);
}

// The block tiles of a solver's hook, up to maxT levels per launch.
HookBlock solver_hook_block(const ps_solver* s, int maxT)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    return hook_block(s->nv, s->ops, maxT, (long long)s->nx * s->ny, sms);
}

// The framework constants of the block tiles (the same for any T).
int hook_block_frame(ps_solver* s, const HookBlock& b)
{
    const int rr = b.rows + 2 * s->ops, cc = kHookBlkW + 2 * s->ops;
    return hook_frame(s, HOOK_STD, rr, cc, s->nv * rr * cc);
}

// A step hook in overlapped blocks.
int run_hook_block(ps_solver* s, const HookBlock& b, int64_t nlevels, int gts0, double* frames,
                   int64_t frame_cap, int frame_every)
{
    const size_t fe = field_elems(s);
    const int its = s->its, every = frame_every > 0 ? frame_every : 1;
    int rc = hook_block_frame(s, b);
    if (rc) return rc;
    for (int64_t done = 0; done < nlevels;) {
        const int64_t left = nlevels - done, k = (left + b.T - 1) / b.T;
        const int T = (int)((left + k - 1) / k);  // even shares
        HookFrames fr = {};
        int any = 0;
        for (int m = 1; m <= T; ++m) {
            const int64_t L = done + m;
            if (!frames || L % its || (L / its) % every || (L / its) / every - 1 >= frame_cap) continue;
            fr.level[m - 1] = at(s, frames, (size_t)((L / its) / every - 1) * fe);
            any = 1;
        }
        double* in = s->base[s->cur];
        double* out = s->base[1 - s->cur];
        if ((rc = timed_launch(s, 5, (double)s->nx * s->ny * T, [&] {
                 hook_block_launch(s, b, T, at(s, in, (size_t)(its - 1) * fe), its == 2 ? in : nullptr,
                                   at(s, out, (size_t)(its - 1) * fe), its == 2 ? out : nullptr, fr,
                                   any, gts0 + (int)done);
             })))
            return rc;
        s->cur = 1 - s->cur;
        done += T;
    }
    return PS_OK;
}

template <bool RK2, class T>
int run_heat_standard(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
                      int frame_every)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
    const double cr = make_params(s).d[0];
    const int rows = standard_rows(s->nx, s->ny, sms);
    const int below = standard_below(RK2, s->nx, s->ny);
    const int grid = standard_grid(s->nx, s->ny, rows, below);
    return run_levels(s, nlevels, gts0, frames, frame_cap, frame_every, 4,
                      [&](const double* cur, const double* prev, double* out, double* fr, int gts) {
                          launch_after(rows == 4 ? heat_standard<RK2, 4, T> : heat_standard<RK2, 8, T>,
                                       grid, 32 * kStdWarps, 0,
                                       s->stream, (const T*)cur, (const T*)prev, (T*)out, (T*)fr,
                                       s->nx, s->ny, gts, cr, below);
                      });
}

int run_swept(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
              int frame_every)
{
    SweptSet K;
    if (s->hook) {
        K = hook_set(s);
    } else if (!pick_swept(s->eq, s->ops, s->its, s->chunk, &K)) {
        return fail(s, PS_ERR_UNSUPPORTED, "no swept kernels for equation %d ops %d its %d chunk %d",
                    s->eq, s->ops, s->its, s->chunk);
    }
    const int O2 = 2 * s->ops;
    const bool fwd_euler = make_params(s).i[0] != 0;
    const bool var = s->eq == PS_EQ_HEATVAR || s->eq == PS_EQ_HEATVAR_ADJMU;
    const bool shape = (s->bs == 16 || s->bs == 32) && s->ny % 32 == 0;
    if (s->dtype == PS_DTYPE_F32 && !(s->eq == PS_EQ_HEAT && s->its == 1 && fwd_euler && shape))
        return fail(s, PS_ERR_UNSUPPORTED,
                    "float32 fields: heat, forward Euler, blocksize 16 or 32, ny a multiple of 32");
    // Column segments of any count up to ny/32 for heat and its
    // variable-courant form on these shapes (they run in blocks of their own
    // size: the count is only reported); divisors of ny for the prisms
    const bool free_seg = s->dtype == PS_DTYPE_F32 ||
                          (shape && s->threads != 256 &&
                           ((s->eq == PS_EQ_HEAT && s->its == 1 && fwd_euler) || var));
    if (s->H < 1 || s->H > s->mpss) return fail(s, PS_ERR_INVALID, "levels per half-cycle %d not in [1, %d]", s->H, s->mpss);
    if (s->chunk < O2 * (s->H + 1))
        return fail(s, PS_ERR_INVALID, "chunk %d narrower than 2*ops*(h+1) = %d", s->chunk, O2 * (s->H + 1));
    if (free_seg) {
        if (s->nseg < 1 || s->nseg > s->ny / 32)
            return fail(s, PS_ERR_INVALID, "nseg %d not in [1, ny/32 = %d]", s->nseg, s->ny / 32);
    } else if (s->nseg < 1 || s->ny % s->nseg) {
        return fail(s, PS_ERR_INVALID, "ny %d not divisible into %d segments", s->ny, s->nseg);
    }
    // the first chunk of a segment shrinks by 2*ops per level on its left edge
    if (!free_seg && std::min(s->chunk, s->ny / s->nseg) < O2 * (s->H + 1))
        return fail(s, PS_ERR_INVALID, "segment width %d narrower than 2*ops*(h+1) = %d",
                    s->ny / s->nseg, O2 * (s->H + 1));
    if (s->nseg_auto) {
        if (free_seg) {
            // as many as 12 warps per SM have bands (8 with a courant number
            // per cell, 16 of 16 rows), of 64 columns or more
            int sms = 148;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
            const int warps = s->bs == 16 ? 16 : (var ? 8 : 12);
            s->nseg = std::max(1, std::min(s->ny / 64, sms * warps / (s->nx / s->bs)));
            s->nseg = std::max(1, std::min(s->nseg, s->ny / 32));
        } else {
            // one CTA per (band, segment): the most segments that divide ny
            // and keep four chunks (and 2*ops*(h+1) columns) each.  Shorter
            // segments make the seams as costly as the streams; longer ones
            // leave few, long CTAs and a ragged last wave.  Measured on Euler
            // (G cell-stages/s): 1024², bs 32: 16 segments 3.00, 8: 3.31,
            // 4: 3.32; 4096², bs 16: 2: 5.65, 16: 6.26, 32: 5.93, 64: 5.39.
            // Step hooks keep eight chunks where that still gives every SM a
            // CTA: their seams are the generic ones, with a slot per level
            // (heat as a hook at 4096², Gcell-updates/s: bs 16, 32 segments
            // 105.5, 16: 113.3; bs 32 at h 6: 128.5 and 135.6).
            int sms = 148;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, s->device);
            int minw = std::max(4 * s->chunk, O2 * (s->H + 1));
            if (s->hook && (s->nx / s->bs) * (s->ny / (8 * s->chunk)) >= sms)
                minw = std::max(minw, 8 * s->chunk);
            s->nseg = 1;
            for (int q = 2; s->ny / q >= minw; ++q)
                if (s->ny % q == 0) s->nseg = q;
        }
    }
    const size_t smem = std::max(stream_smem(s), seam_smem(s));
    if (smem > 227 * 1024)
        return fail(s, PS_ERR_UNSUPPORTED, "tile needs %zu bytes of shared memory", smem);
    // heat in overlapped blocks; threads 256 keeps the shared-memory prisms
    // (float64), and a configured h bounds the levels of a launch
    if (!s->hook && s->eq == PS_EQ_HEAT && (s->threads != 256 || s->dtype == PS_DTYPE_F32) &&
        (s->its == 1) == fwd_euler) {
        const int maxT = s->h_set ? s->H : kTileMaxT;
        if (s->dtype == PS_DTYPE_F32)
            return run_block<float, false>(s, nlevels, gts0, frames, frame_cap, frame_every, maxT);
        if (fwd_euler)
            return run_block<double, false>(s, nlevels, gts0, frames, frame_cap, frame_every, maxT);
        // (frames that 4-wide stores cannot reach may fall on half stages)
        if (maxT >= 2 && aligned32(frames))
            return run_block<double, true>(s, nlevels, gts0, frames, frame_cap, frame_every, maxT);
    }
    if (s->hook && s->threads != 256) {
        const HookBlock b = solver_hook_block(s, s->h_set ? s->H : kHookBlkMaxT);
        if (b.rows) return run_hook_block(s, b, nlevels, gts0, frames, frame_cap, frame_every);
    }
    if (s->eq == PS_EQ_EULER && s->threads != 256)
        return run_march(s, nlevels, gts0, frames, frame_cap, frame_every, 5);
    if (s->threads != 256) {
        if (s->eq == PS_EQ_HEATVAR && !s->field[1])
            return run_var<VAR_FORWARD>(s, nlevels, gts0, frames, frame_cap, frame_every);
        if (s->eq == PS_EQ_HEATVAR)
            return run_var<VAR_RECOMPUTE>(s, nlevels, gts0, frames, frame_cap, frame_every);
        if (s->eq == PS_EQ_HEATVAR_ADJ)
            return run_var<VAR_LAMBDA>(s, nlevels, gts0, frames, frame_cap, frame_every);
        if (s->eq == PS_EQ_HEATVAR_ADJMU)
            return run_var<VAR_MU>(s, nlevels, gts0, frames, frame_cap, frame_every);
    }
    int rc = ensure_swept_buffers(s);
    if (rc) return rc;
    if (!s->side) {
        int lo = 0, hi = 0;
        PS_CUDA(s, cudaDeviceGetStreamPriorityRange(&lo, &hi));
        PS_CUDA(s, cudaStreamCreateWithPriority(&s->side, cudaStreamNonBlocking, hi));
        PS_CUDA(s, cudaEventCreateWithFlags(&s->ev_fork, cudaEventDisableTiming));
        PS_CUDA(s, cudaEventCreateWithFlags(&s->ev_join, cudaEventDisableTiming));
    }
    SweptArgs a;
    memset(&a, 0, sizeof a);
    a.frames = frames;
    a.frame_cap = frames ? frame_cap : 0;
    a.frame_every = frame_every > 0 ? frame_every : 1;
    a.nx = s->nx;
    a.ny = s->ny;
    a.nv = s->nv;
    a.bx = s->bs;
    a.hx = s->bs / 2;
    a.Hmax = s->H;
    a.nb = s->nx / s->bs;
    a.nseg = s->nseg;
    a.wy = s->ny / a.nseg;
    a.nchunks = (a.wy + s->chunk - 1) / s->chunk;  // the last chunk may be partial
    a.seg_unit = a.wy;
    a.seg_units = a.nseg;
    a.its = s->its;
    a.gts_base = gts0 - 1;
    a.xface = s->xface;
    a.yface = s->yface;
    a.p = make_params(s);
    a.seam_direct = solver_seam_direct(s) ? 1 : 0;
    const int units = a.nb * a.nseg;
    if (s->hook) {
        // the hook's tiles: stream slots of bs rows x (chunk + 2 OPS) columns
        // whose levels sit one slot + OPS apart (the chunk's parallelogram),
        // seam slots of bs rows x 2 OPS (Hmax + 1) columns, one slot apart
        const int rs = s->chunk + O2, tw = 2 * s->ops * (s->H + 1);
        if ((rc = hook_frame(s, HOOK_STREAM, s->bs, rs, s->nv * s->bs * rs + s->ops)) ||
            (rc = hook_frame(s, HOOK_SEAM, s->bs, tw, s->nv * s->bs * tw)))
            return rc;
    }
    const size_t fe = field_elems(s);
    int off = 0;
    int64_t done = 0;
    while (done < nlevels) {
        const int H = (int)std::min<int64_t>(s->H, nlevels - done);
        a.H = H;
        a.L0 = done;
        a.off = off;
        a.bin = s->base[s->cur];
        a.bout = s->base[1 - s->cur];
        if (H < s->its) {
            // the newest its-H base levels carry over unchanged
            for (int q = 0; q < s->its - H; ++q)
                PS_CUDA(s, cudaMemcpyAsync(at(s, s->base[1 - s->cur], (size_t)q * fe),
                                           at(s, s->base[s->cur], (size_t)(q + H) * fe),
                                           nbytes(s, fe), cudaMemcpyDeviceToDevice, s->stream));
        }
        // algorithmic cell updates of each kernel in this half-cycle
        double cP = 0, cY = 0, cG = 0, cO = 0;
        for (int m = 1; m <= H; ++m) {
            const double rp = s->bs - 2.0 * s->ops * m, rg = 2.0 * s->ops * m;
            const double cm = 2.0 * s->ops * m * s->nseg;  // seam columns of a band
            const double cs = (double)s->ny - cm;           // stream columns of a band
            cP += rp * cs;
            cY += rp * cm;
            cG += rg * cs;
            cO += rg * cm;
        }
        const double u = (double)a.nb;
        const size_t psm = stream_smem(s);
        // P, then Y on `stream` beside G on the side stream (G reads nothing
        // that Y writes: its valid cells depend on the prisms' faces only,
        // and adjacent bands share their segment boundaries, so G's
        // trapezoids avoid both bands' y-bridge diamonds; it writes its
        // y-faces into the second buffer), then O
        SweptArgs ag = a;
        ag.yface = at(s, s->yface, s->yface_n / 2);
        if ((rc = timed_launch(s, 0, cP * u, [&] { K.P(a, units, psm, s->stream); }))) return rc;
        PS_CUDA(s, cudaEventRecord(s->ev_fork, s->stream));
        PS_CUDA(s, cudaStreamWaitEvent(s->side, s->ev_fork, 0));
        if ((rc = timed_launch(s, 2, cG * u, [&] { K.G(ag, units, psm, s->side); }, s->side))) return rc;
        PS_CUDA(s, cudaEventRecord(s->ev_join, s->side));
        if ((rc = timed_launch(s, 1, cY * u, [&] { K.Y(a, units, seam_smem(s), s->stream); }))) return rc;
        PS_CUDA(s, cudaStreamWaitEvent(s->stream, s->ev_join, 0));
        if ((rc = timed_launch(s, 3, cO * u, [&] { K.O(ag, units, seam_smem(s), s->stream); }))) return rc;
        s->cur = 1 - s->cur;
        off = ((off - a.hx) % s->nx + s->nx) % s->nx;
        done += H;
    }
    return PS_OK;
}

int run_standard(ps_solver* s, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
                 int frame_every)
{
    StdLaunch K = s->hook ? nullptr : pick_standard(s->eq, s->ops);
    if (!K && !s->hook) return fail(s, PS_ERR_UNSUPPORTED, "no standard kernel for equation %d", s->eq);
    // (threads = 256 keeps the per-cell kernels)
    if (s->eq == PS_EQ_EULER && s->threads != 256)
        return run_march(s, nlevels, gts0, frames, frame_cap, frame_every, 4);
    if (s->eq == PS_EQ_HEAT && s->threads != 256) {
        const bool fwd = make_params(s).i[0] != 0;
        if (s->dtype == PS_DTYPE_F32) {
            if (fwd && s->ny % 64 == 0)
                return run_heat_standard<false, float>(s, nlevels, gts0, frames, frame_cap, frame_every);
        } else if (fwd) {
            return run_heat_standard<false, double>(s, nlevels, gts0, frames, frame_cap, frame_every);
        } else if (s->its == 2) {
            return run_heat_standard<true, double>(s, nlevels, gts0, frames, frame_cap, frame_every);
        }
    }
    if (s->dtype == PS_DTYPE_F32)
        return fail(s, PS_ERR_UNSUPPORTED,
                    "float32 fields: heat with forward Euler and ny a multiple of 64 only");
    const size_t fe = field_elems(s);
    for (int i = 0; i < 3; ++i)
        if (!s->ring[i]) PS_CUDA(s, cudaMalloc(&s->ring[i], nbytes(s, fe)));
    const int its = s->its;
    // ring[c] = current level, ring[p] = previous level
    int c = 0, p = 1, n = 2;
    double* b = s->base[s->cur];
    PS_CUDA(s, cudaMemcpyAsync(s->ring[c], at(s, b, (size_t)(its - 1) * fe), nbytes(s, fe),
                               cudaMemcpyDeviceToDevice, s->stream));
    PS_CUDA(s, cudaMemcpyAsync(s->ring[p], at(s, b, (size_t)(its >= 2 ? its - 2 : 0) * fe),
                               nbytes(s, fe), cudaMemcpyDeviceToDevice, s->stream));
    const EqParams prm = make_params(s);
    const int every = frame_every > 0 ? frame_every : 1;
    int rc;
    HookBlock blk{};
    if (s->hook) {
        blk = solver_hook_block(s, 1);
        if (!blk.rows) return fail(s, PS_ERR_UNSUPPORTED, "the hook's standard tile does not fit in shared memory");
        if ((rc = hook_block_frame(s, blk))) return rc;
    }
    for (int64_t L = 1; L <= nlevels; ++L) {
        double* fr = nullptr;
        if (frames && L % its == 0 && (L / its) % every == 0) {
            const int64_t slot = (L / its) / every - 1;
            if (slot < frame_cap) fr = at(s, frames, (size_t)slot * fe);
        }
        const int gts = gts0 + (int)(L - 1);
        if ((rc = timed_launch(s, 4, (double)s->nx * s->ny, [&] {
                 if (s->hook) {
                     HookFrames f = {};
                     f.level[0] = fr;
                     hook_block_launch(s, blk, 1, s->ring[c], s->ring[p], s->ring[n], nullptr, f, fr != nullptr, gts);
                 } else {
                     K(s->ring[c], s->ring[p], s->ring[n], fr, s->nx, s->ny, s->nv, gts, prm,
                       s->stream);
                 }
             })))
            return rc;
        const int t = p;
        p = c;
        c = n;
        n = t;
    }
    // newest levels back into the base
    PS_CUDA(s, cudaMemcpyAsync(at(s, b, (size_t)(its - 1) * fe), s->ring[c], nbytes(s, fe),
                               cudaMemcpyDeviceToDevice, s->stream));
    if (its >= 2)
        PS_CUDA(s, cudaMemcpyAsync(at(s, b, (size_t)(its - 2) * fe), s->ring[p], nbytes(s, fe),
                                   cudaMemcpyDeviceToDevice, s->stream));
    return PS_OK;
}

struct GlobalSpec {
    const char* name;
    int eqmask;  // bit per equation
};

const GlobalSpec kGlobals[] = {
    {"DT", 0x1f},    {"DX", 0x1f},      {"DY", 0x1f},   {"ALPHA", 1 << PS_EQ_HEAT},
    {"SCHEME", (1 << PS_EQ_HEAT) | (1 << PS_EQ_EXAMPLE) | (1 << PS_EQ_CHECKER)},
    {"GAMMA", 1 << PS_EQ_EULER}, {"GAM_M1", 1 << PS_EQ_EULER}, {"DTDX", 1 << PS_EQ_EULER},
    {"DTDY", 1 << PS_EQ_EULER}, {"LEN", (1 << PS_EQ_HEATVAR) | (1 << PS_EQ_HEATVAR_ADJ) | (1 << PS_EQ_HEATVAR_ADJMU)},
};

const GlobalSpec* find_global(const ps_solver* s, const char* name)
{
    for (const auto& g : kGlobals)
        if (!strcmp(g.name, name) && (g.eqmask >> s->eq & 1)) return &g;
    return nullptr;
}

double decode_value(const void* value, size_t nbytes)
{
    switch (nbytes) {
    case 8: {
        double d;
        memcpy(&d, value, 8);
        return d;
    }
    case 4: {
        int32_t i;
        memcpy(&i, value, 4);
        return (double)i;
    }
    case 2: {
        int16_t i;
        memcpy(&i, value, 2);
        return (double)i;
    }
    case 1: return (double)*(const uint8_t*)value;
    default: return 0.0;
    }
}

int solver_open(ps_solver* s);

// Kind of a hook constant, from its declaration in the hook's source:
// 'f' floating point, 'b' bool, 'i' any other (integer) type.
char hook_const_kind(const std::string& src, const std::string& name)
{
    size_t pos = 0;
    while ((pos = src.find("__constant__", pos)) != std::string::npos) {
        const size_t end = src.find(';', pos);
        if (end == std::string::npos) break;
        const std::string decl = src.substr(pos, end - pos);
        pos = end;
        // the name as a whole word of the declaration
        size_t k = 0;
        bool found = false;
        while ((k = decl.find(name, k)) != std::string::npos) {
            const bool l = k == 0 || !(isalnum((unsigned char)decl[k - 1]) || decl[k - 1] == '_');
            const size_t e = k + name.size();
            const bool r = e >= decl.size() || !(isalnum((unsigned char)decl[e]) || decl[e] == '_');
            if (l && r) {
                found = true;
                break;
            }
            k = e;
        }
        if (!found) continue;
        if (decl.find("double") != std::string::npos || decl.find("float") != std::string::npos)
            return 'f';
        if (decl.find("bool") != std::string::npos) return 'b';
        return 'i';
    }
    return 'f';
}

// The value in the representation of a hook constant of `size` bytes and
// `kind` (the caller's bytes as they are when the sizes agree, else converted
// through double).
bool hook_encode(const void* value, size_t nbytes, size_t size, char kind, unsigned char* buf)
{
    if (nbytes == size) {
        memcpy(buf, value, size);
        return true;
    }
    const double d = decode_value(value, nbytes);
    if (kind == 'f' && size == 8) {
        memcpy(buf, &d, 8);
    } else if (kind == 'f' && size == 4) {
        const float f = (float)d;
        memcpy(buf, &f, 4);
    } else if (size == 8) {
        const int64_t i = (int64_t)d;
        memcpy(buf, &i, 8);
    } else if (size == 4) {
        const int32_t i = (int32_t)d;
        memcpy(buf, &i, 4);
    } else if (size == 2) {
        const int16_t i = (int16_t)d;
        memcpy(buf, &i, 2);
    } else if (size == 1) {
        buf[0] = kind == 'b' ? (d != 0.0) : (unsigned char)(int)d;
    } else {
        return false;
    }
    return true;
}

}  // namespace

// Maps the pages of a host buffer about to receive n bytes, in one call, while
// the GPU may still be busy.  A fresh allocation otherwise takes a page fault
// every 4 KB of the copy: 25 MB in 25 arrays, 10 ms by faults, 5 ms here, the copy
// itself 2.  Looks at one page only where they are mapped already.  Advice: the
// copy works whatever becomes of it.
static void map_host_pages(void* p, size_t n)
{
#ifdef MADV_POPULATE_WRITE
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const uintptr_t lo = ((uintptr_t)p + page - 1) / page * page, hi = ((uintptr_t)p + n) / page * page;
    if (hi < lo + 16 * page) return;
    unsigned char there = 1;
    const uintptr_t mid = (lo + (hi - lo) / 2) / page * page;
    if (mincore((void*)mid, page, &there) == 0 && !(there & 1))
        madvise((void*)lo, hi - lo, MADV_POPULATE_WRITE);
#else
    (void)p;
    (void)n;
#endif
}

extern "C" {

const char* ps_version(void) { return kVersion; }

const char* ps_last_error(const ps_solver* s)
{
    return s ? s->err.c_str() : g_create_error.c_str();
}

int64_t ps_kernel_launches(const ps_solver* s) { return s ? s->launches : 0; }

int ps_create(ps_solver** out, int device, int equation, int nv, int nx, int ny, int ops, int its,
              int blocksize)
{
    return ps_create_typed(out, device, equation, nv, nx, ny, ops, its, blocksize, PS_DTYPE_F64);
}

int ps_create_typed(ps_solver** out, int device, int equation, int nv, int nx, int ny, int ops,
                    int its, int blocksize, int dtype)
{
    if (!out) return PS_ERR_INVALID;
    *out = nullptr;
    if (equation < PS_EQ_HEAT || equation > PS_EQ_HEATVAR_ADJMU || equation == PS_EQ_HOOK)
        return PS_ERR_INVALID;
    if (dtype != PS_DTYPE_F64 && dtype != PS_DTYPE_F32) return PS_ERR_INVALID;
    ps_solver* s = new ps_solver();
    s->dtype = dtype;
    s->esize = dtype == PS_DTYPE_F32 ? sizeof(float) : sizeof(double);
    s->device = device;
    s->eq = equation;
    s->nv = nv;
    s->nx = nx;
    s->ny = ny;
    s->ops = eq_ops(equation, ops);
    s->its = its;
    s->bs = blocksize;
    int rc = PS_OK;
    if (equation == PS_EQ_HEAT || equation == PS_EQ_HALF) {
        if (nv != 1) rc = fail(s, PS_ERR_INVALID, "heat/half have one variable, got nv=%d", nv);
    }
    if (((equation == PS_EQ_HEATVAR || equation == PS_EQ_HEATVAR_ADJMU) && nv != 1) ||
        (equation == PS_EQ_HEATVAR_ADJ && nv != 2) ||
        ((equation == PS_EQ_HEATVAR || equation == PS_EQ_HEATVAR_ADJ || equation == PS_EQ_HEATVAR_ADJMU) &&
         its != 1))
        rc = fail(s, PS_ERR_INVALID,
                  "heatvar and its mu-form adjoint have nv=1, the lambda-form adjoint nv=2; its=1 "
                  "(got nv=%d its=%d)", nv, its);
    if (equation == PS_EQ_EULER && (nv != 4 || its != 2))
        rc = fail(s, PS_ERR_INVALID, "euler needs nv=4 and its=2 (got nv=%d its=%d)", nv, its);
    if (ops != s->ops) rc = fail(s, PS_ERR_INVALID, "equation %d has ops=%d, got %d", equation, s->ops, ops);
    if (dtype == PS_DTYPE_F32 && (equation != PS_EQ_HEAT || its != 1))
        rc = fail(s, PS_ERR_UNSUPPORTED, "float32 fields: heat with forward Euler (its=1) only");
    if (nv < 1 || nv > 4 || its < 1 || its > 2 || ops < 1 || ops > 2)
        rc = fail(s, PS_ERR_UNSUPPORTED, "nv in 1..4, its in 1..2, ops in 1..2 supported");
    if (blocksize <= 0 || blocksize % (2 * s->ops))  // io.py:52
        rc = fail(s, PS_ERR_INVALID, "blocksize %d must be a multiple of 2*ops", blocksize);
    if (rc == PS_OK && (nx % blocksize || ny % blocksize))  // process.py:143
        rc = fail(s, PS_ERR_INVALID, "array %dx%d not divisible by blocksize %d", nx, ny, blocksize);
    if (rc == PS_OK && (size_t)3 * nv * nx * ny >= (size_t)1 << 31)
        rc = fail(s, PS_ERR_UNSUPPORTED, "field too large for 32-bit offsets");
    s->mpss = blocksize / (2 * s->ops) - 1;
    if (rc == PS_OK && s->mpss < 1)
        rc = fail(s, PS_ERR_INVALID, "blocksize %d gives no swept level (MPSS < 1)", blocksize);
    s->H = default_levels(s->eq, s->its, blocksize, s->mpss);
    s->chunk = (2 * s->ops * (s->H + 1) <= 32) ? 32 : 64;
    // Euler: 64-column chunks keep every thread of a stream CTA busy on each
    // level, where the tile fits in shared memory
    if (s->eq == PS_EQ_EULER && s->chunk == 32) {
        s->chunk = 64;
        if (stream_smem(s) > 227 * 1024) s->chunk = 32;
    }
    if (rc == PS_OK) rc = solver_open(s);
    if (rc != PS_OK) {
        g_create_error = s->err;  // readable through ps_last_error(NULL)
        ps_destroy(s);
        return rc;
    }
    *out = s;
    return PS_OK;
}

}  // extern "C"

namespace {

// The device half of solver creation: device, stream, base buffers.
int solver_open(ps_solver* s)
{
    const int device = s->device, nv = s->nv, nx = s->nx, ny = s->ny, its = s->its;
    int rc = PS_OK;
    s->nseg = 1;
    if (rc == PS_OK) {
        cudaError_t e = cudaSetDevice(device);
        if (e != cudaSuccess) rc = fail(s, PS_ERR_CUDA, "cudaSetDevice: %s", cudaGetErrorString(e));
    }
    if (rc == PS_OK) {
        cudaError_t e = cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) rc = fail(s, PS_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e));
        s->own_stream = true;
    }
    if (rc == PS_OK) {
        const size_t bytes = nbytes(s, (size_t)its * nv * nx * ny);
        for (int i = 0; i < 2 && rc == PS_OK; ++i) {
            cudaError_t e = cudaMalloc(&s->base[i], bytes);
            if (e != cudaSuccess) rc = fail(s, PS_ERR_NOMEM, "cudaMalloc base: %s", cudaGetErrorString(e));
        }
    }
    return rc;
}

}  // namespace

extern "C" {

int ps_hook_check(const char* source, const char* name, int nv, int ops, int its, char* log,
                  size_t loglen)
{
    if (log && loglen) log[0] = '\0';
    if (!source || nv < 1 || nv > 8 || ops < 1 || ops > 4 || its < 1 || its > 2)
        return PS_ERR_INVALID;
    std::vector<char> cubin;
    std::string lg;
    const int rc = hook_compile(hook_program(source, name ? name : "hook.cu", nv, ops, its), &cubin, &lg);
    if (log && loglen) {
        strncpy(log, lg.c_str(), loglen - 1);
        log[loglen - 1] = '\0';
    }
    return rc;
}

int ps_create_hook(ps_solver** out, int device, const char* source, const char* name, int nv,
                   int nx, int ny, int ops, int its, int blocksize)
{
    if (!out) return PS_ERR_INVALID;
    *out = nullptr;
    ps_solver* s = new ps_solver();
    s->device = device;
    s->eq = PS_EQ_HOOK;
    s->nv = nv;
    s->nx = nx;
    s->ny = ny;
    s->ops = ops;
    s->its = its;
    s->bs = blocksize;
    int rc = PS_OK;
    if (!source) rc = fail(s, PS_ERR_INVALID, "no hook source");
    else if (nv < 1 || nv > 8 || ops < 1 || ops > 4 || its < 1 || its > 2)
        rc = fail(s, PS_ERR_UNSUPPORTED, "step hooks: nv in 1..8, ops in 1..4, its in 1..2");
    else if (blocksize <= 0 || blocksize % (2 * ops))  // io.py:52
        rc = fail(s, PS_ERR_INVALID, "blocksize %d must be a multiple of 2*ops", blocksize);
    else if (nx <= 0 || ny <= 0 || nx % blocksize || ny % blocksize)  // process.py:143
        rc = fail(s, PS_ERR_INVALID, "array %dx%d not divisible by blocksize %d", nx, ny, blocksize);
    else if ((size_t)3 * nv * nx * ny >= (size_t)1 << 31)
        rc = fail(s, PS_ERR_UNSUPPORTED, "field too large for 32-bit offsets");
    s->mpss = blocksize > 0 && ops > 0 ? blocksize / (2 * ops) - 1 : 0;
    if (rc == PS_OK && s->mpss < 1)
        rc = fail(s, PS_ERR_INVALID, "blocksize %d gives no swept level (MPSS < 1)", blocksize);
    if (rc == PS_OK) {
        s->hook = new HookModule();
        s->hook->nv = nv;
        s->hook->ops = ops;
        s->hook->its = its;
        s->hook_src = source;
        // levels per half-cycle: the most (up to MPSS) whose stream tile,
        // one linear slot per level, leaves room for three CTAs per SM; where
        // none does, the most that fit at all.  (The heat plugin as a hook,
        // 4096², 600 steps, Gcell-updates/s: bs 32 at MPSS = 15, one CTA per
        // SM, 59; at 6, three CTAs, 136; bs 16 keeps MPSS = 7.)
        for (const size_t cap : {(size_t)227 * 1024 / 3, (size_t)227 * 1024}) {
            s->H = s->mpss;
            bool fits = false;
            for (;;) {
                s->chunk = (2 * ops * (s->H + 1) <= 32) ? 32 : 64;
                fits = 2 * ops * (s->H + 1) <= 64 && stream_smem(s) <= cap &&
                       seam_smem(s) <= 227 * 1024;
                if (fits || s->H == 1) break;
                --s->H;
            }
            if (fits) break;
        }
        std::vector<char> cubin;
        std::string log;
        rc = hook_compile(hook_program(source, name ? name : "hook.cu", nv, ops, its), &cubin, &log);
        if (rc) fail(s, PS_ERR_COMPILE, "step hook %s did not compile:\n%s", name ? name : "", log.c_str());
        if (rc == PS_OK) rc = solver_open(s);  // device, stream (the primary context), bases
        if (rc == PS_OK) {
            std::string err;
            if (hook_load(s->hook, cubin, &err)) rc = fail(s, PS_ERR_CUDA, "%s", err.c_str());
        }
    }
    if (rc != PS_OK) {
        g_create_error = s->err;
        ps_destroy(s);
        return rc;
    }
    *out = s;
    return PS_OK;
}

int ps_destroy(ps_solver* s)
{
    if (!s) return PS_OK;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    for (auto& b : s->base)
        if (b) cudaFree(b);
    for (auto& r : s->ring)
        if (r) cudaFree(r);
    if (s->xface) cudaFree(s->xface);
    if (s->yface) cudaFree(s->yface);
    if (s->hook) {
        if (s->hook->mod) drv().moduleUnload(s->hook->mod);
        delete s->hook;
    }
    for (auto& p : s->pending) {
        cudaEventDestroy(p.second.first);
        cudaEventDestroy(p.second.second);
    }
    for (auto e : s->event_pool) cudaEventDestroy(e);
    if (s->side) {
        cudaStreamSynchronize(s->side);
        cudaStreamDestroy(s->side);
    }
    if (s->ev_fork) cudaEventDestroy(s->ev_fork);
    if (s->ev_join) cudaEventDestroy(s->ev_join);
    if (s->own_stream && s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return PS_OK;
}

int ps_set_global(ps_solver* s, const char* name, const void* value, size_t nbytes)
{
    if (!s || !name || !value) return PS_ERR_INVALID;
    if (nbytes != 1 && nbytes != 2 && nbytes != 4 && nbytes != 8)
        return fail(s, PS_ERR_INVALID, "constant %s: unsupported size %zu", name, nbytes);
    if (s->hook) {
        // the hook's own __constant__, in every kernel kind's copy, written in
        // stream order (kernels queued before keep the old value)
        PS_CUDA(s, cudaSetDevice(s->device));
        HookConst* c = hook_const(s->hook, name);
        if (!c) return fail(s, PS_ERR_INVALID, "the step hook declares no __constant__ %s", name);
        unsigned char buf[8];
        if (!hook_encode(value, nbytes, c->size, hook_const_kind(s->hook_src, name), buf))
            return fail(s, PS_ERR_UNSUPPORTED, "constant %s: %zu-byte type", name, c->size);
        for (int k = 0; k < 3; ++k) {
            CUresult r = drv().memcpyHtoDAsync(c->ptr[k], buf, c->size, (CUstream)s->stream);
            if (r != CUDA_SUCCESS)
                return fail(s, PS_ERR_CUDA, "constant %s: %s", name, cu_error(r).c_str());
        }
        s->globals[name] = decode_value(value, nbytes);
        return PS_OK;
    }
    if (!find_global(s, name)) return fail(s, PS_ERR_INVALID, "no constant named %s", name);
    s->globals[name] = decode_value(value, nbytes);
    return PS_OK;
}

int ps_get_global(ps_solver* s, const char* name, void** handle, size_t* size)
{
    if (!s || !name) return PS_ERR_INVALID;
    if (s->hook) {
        PS_CUDA(s, cudaSetDevice(s->device));
        HookConst* c = hook_const(s->hook, name);
        if (!c) return fail(s, PS_ERR_INVALID, "the step hook declares no __constant__ %s", name);
        if (handle) *handle = (void*)c;  // `name` first, like the built-ins' GlobalSpec
        if (size) *size = c->size;
        return PS_OK;
    }
    const GlobalSpec* g = find_global(s, name);
    if (!g) return fail(s, PS_ERR_INVALID, "no constant named %s", name);
    if (handle) *handle = (void*)g;
    if (size) *size = !strcmp(name, "SCHEME") ? 4 : 8;
    return PS_OK;
}

int ps_set_global_handle(ps_solver* s, void* handle, const void* value, size_t nbytes)
{
    if (!s || !handle) return PS_ERR_INVALID;
    return ps_set_global(s, ((const GlobalSpec*)handle)->name, value, nbytes);
}

int ps_get_global_value(ps_solver* s, const char* name, double* value)
{
    if (!s || !name || !value) return PS_ERR_INVALID;
    const int SX = s->nx, SY = s->ny;
    const int T = 2 * s->mpss + s->its;
    if (!strcmp(name, "NV")) *value = s->nv;
    else if (!strcmp(name, "SX")) *value = SX;
    else if (!strcmp(name, "SY")) *value = SY;
    else if (!strcmp(name, "VARS")) *value = (double)SX * SY;
    else if (!strcmp(name, "TIMES")) *value = (double)s->nv * SX * SY;
    else if (!strcmp(name, "MPSS")) *value = s->mpss;
    else if (!strcmp(name, "MOSS")) *value = 2 * s->mpss;
    else if (!strcmp(name, "OPS")) *value = s->ops;
    else if (!strcmp(name, "ITS")) *value = s->its;
    else if (!strcmp(name, "T")) *value = T;
    else {
        auto it = s->globals.find(name);
        if (it == s->globals.end()) return fail(s, PS_ERR_INVALID, "no constant named %s", name);
        *value = it->second;
    }
    return PS_OK;
}

int ps_configure(ps_solver* s, int h, int nseg, int chunk, int threads)
{
    if (!s) return PS_ERR_INVALID;
    if (h < 0 || nseg < 0 || chunk < 0 || threads < 0) return fail(s, PS_ERR_INVALID, "negative knob");
    if (h) {
        if (h > s->mpss) return fail(s, PS_ERR_INVALID, "h %d > MPSS %d", h, s->mpss);
        s->H = h;
        s->h_set = true;
    }
    if (nseg) {
        s->nseg = nseg;
        s->nseg_auto = false;
    }
    if (chunk) {
        if (chunk != 32 && chunk != 64) return fail(s, PS_ERR_INVALID, "chunk must be 32 or 64");
        s->chunk = chunk;
    }
    if (threads) {
        // 128: overlapped blocks and level-by-level kernels where they apply
        // (default); 256: always the shared-memory prisms
        if (threads != 256 && threads != 128)
            return fail(s, PS_ERR_UNSUPPORTED, "threads must be 128 or 256");
        s->threads = threads;
    }
    return PS_OK;
}

int ps_get_tiling(ps_solver* s, int* h, int* nseg, int* chunk, int* mpss)
{
    if (!s) return PS_ERR_INVALID;
    if (h) *h = s->H;
    if (nseg) *nseg = s->nseg;
    if (chunk) *chunk = s->chunk;
    if (mpss) *mpss = s->mpss;
    return PS_OK;
}

int ps_set_state(ps_solver* s, const double* src, int levels, int src_on_device)
{
    if (!s || !src) return PS_ERR_INVALID;
    if (levels != 1 && levels != s->its)
        return fail(s, PS_ERR_INVALID, "levels must be 1 or its=%d", s->its);
    PS_CUDA(s, cudaSetDevice(s->device));
    const size_t fe = field_elems(s);
    const cudaMemcpyKind kind = src_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    for (int q = 0; q < s->its; ++q) {
        const double* from = at(s, const_cast<double*>(src), (size_t)(levels == 1 ? 0 : q) * fe);
        PS_CUDA(s, cudaMemcpyAsync(at(s, s->base[s->cur], (size_t)q * fe), from, nbytes(s, fe),
                                   kind, s->stream));
    }
    if (!src_on_device) PS_CUDA(s, cudaStreamSynchronize(s->stream));
    s->have_state = true;
    return PS_OK;
}

int ps_set_field(ps_solver* s, int index, double* d_field)
{
    if (!s) return PS_ERR_INVALID;
    if (s->eq != PS_EQ_HEATVAR && s->eq != PS_EQ_HEATVAR_ADJ && s->eq != PS_EQ_HEATVAR_ADJMU)
        return fail(s, PS_ERR_INVALID, "equation %d reads no grid fields", s->eq);
    if (index < 0 || index > 2) return fail(s, PS_ERR_INVALID, "field index %d not 0, 1 or 2", index);
    s->field[index] = d_field;
    return PS_OK;
}

int ps_run(ps_solver* s, int mode, int64_t nlevels, int gts0, double* frames, int64_t frame_cap,
           int frame_every, int frames_on_device)
{
    if (!s) return PS_ERR_INVALID;
    if (!s->have_state) return fail(s, PS_ERR_STATE, "ps_run before ps_set_state");
    if (nlevels < 0) return fail(s, PS_ERR_INVALID, "negative level count");
    if (frame_every < 0) return fail(s, PS_ERR_INVALID, "negative frame_every");
    const bool hv = s->eq == PS_EQ_HEATVAR || s->eq == PS_EQ_HEATVAR_ADJ || s->eq == PS_EQ_HEATVAR_ADJMU;
    if (hv && !s->field[0]) return fail(s, PS_ERR_STATE, "heatvar: no courant field (ps_set_field 0)");
    if ((s->eq == PS_EQ_HEATVAR_ADJ || s->eq == PS_EQ_HEATVAR_ADJMU) && !s->field[1])
        return fail(s, PS_ERR_STATE, "heatvar adjoint: no recomputed Laplacians (ps_set_field 1)");
    if (s->eq == PS_EQ_HEATVAR_ADJMU && !s->field[2])
        return fail(s, PS_ERR_STATE, "heatvar adjoint (mu): no sum field (ps_set_field 2)");
    if (hv && s->field[1] && nlevels > 0) {
        // field 1 holds LEN levels: the run's levels gts0 .. gts0+nlevels-1 must index them
        auto it = s->globals.find("LEN");
        const int64_t len = it == s->globals.end() ? 0 : (int64_t)it->second;
        if (gts0 < 1 || gts0 - 1 + nlevels > len)
            return fail(s, PS_ERR_INVALID, "levels %d..%lld outside the %lld levels of field 1 (LEN)",
                        gts0, (long long)(gts0 - 1 + nlevels), (long long)len);
    }
    PS_CUDA(s, cudaSetDevice(s->device));
    double* dframes = frames;
    const size_t fe = field_elems(s);
    if (frames && !frames_on_device) {
        if (frame_cap > 0) PS_CUDA(s, cudaMallocAsync(&dframes, nbytes(s, (size_t)frame_cap * fe), s->stream));
        else dframes = nullptr;
    }
    int rc;
    if (mode == PS_MODE_SWEPT) rc = run_swept(s, nlevels, gts0, dframes, frame_cap, frame_every);
    else if (mode == PS_MODE_STANDARD) rc = run_standard(s, nlevels, gts0, dframes, frame_cap, frame_every);
    else rc = fail(s, PS_ERR_INVALID, "mode %d", mode);
    if (frames && !frames_on_device && dframes) {
        if (rc == PS_OK)
            PS_CUDA(s, cudaMemcpyAsync(frames, dframes, nbytes(s, (size_t)frame_cap * fe),
                                       cudaMemcpyDeviceToHost, s->stream));
        cudaFreeAsync(dframes, s->stream);
        PS_CUDA(s, cudaStreamSynchronize(s->stream));
    }
    return rc;
}

int ps_get_state(ps_solver* s, double* dst, int level, int dst_on_device)
{
    if (!s || !dst) return PS_ERR_INVALID;
    if (level < 0 || level >= s->its) return fail(s, PS_ERR_INVALID, "level %d not in [0, its)", level);
    PS_CUDA(s, cudaSetDevice(s->device));
    const size_t fe = field_elems(s);
    if (!dst_on_device) map_host_pages(dst, nbytes(s, fe));
    PS_CUDA(s, cudaMemcpyAsync(dst, at(s, s->base[s->cur], (size_t)(s->its - 1 - level) * fe),
                               nbytes(s, fe),
                               dst_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                               s->stream));
    if (!dst_on_device) PS_CUDA(s, cudaStreamSynchronize(s->stream));
    return PS_OK;
}

// rows [row0, row0+nrows) of every variable of one base level <-> a packed
// [nv][nrows][ny] buffer: one strided copy (variables are nx*ny apart)
static int rows_copy(ps_solver* s, int level, int row0, int nrows, double* buf, int on_device,
                     bool to_buf)
{
    if (!s || !buf) return PS_ERR_INVALID;
    if (level < 0 || level >= s->its) return fail(s, PS_ERR_INVALID, "level %d not in [0, its)", level);
    if (row0 < 0 || nrows < 0 || row0 + nrows > s->nx)
        return fail(s, PS_ERR_INVALID, "rows [%d, %d) outside [0, %d)", row0, row0 + nrows, s->nx);
    if (nrows == 0) return PS_OK;
    PS_CUDA(s, cudaSetDevice(s->device));
    const size_t fe = field_elems(s), plane = (size_t)s->nx * s->ny;
    double* f = at(s, s->base[s->cur], (size_t)(s->its - 1 - level) * fe + (size_t)row0 * s->ny);
    const size_t width = nbytes(s, (size_t)nrows * s->ny);
    if (to_buf)
        PS_CUDA(s, cudaMemcpy2DAsync(buf, width, f, nbytes(s, plane), width, s->nv,
                                     on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                     s->stream));
    else
        PS_CUDA(s, cudaMemcpy2DAsync(f, nbytes(s, plane), buf, width, width, s->nv,
                                     on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                                     s->stream));
    if (!on_device) PS_CUDA(s, cudaStreamSynchronize(s->stream));
    return PS_OK;
}

int ps_get_rows(ps_solver* s, int level, int row0, int nrows, double* dst, int dst_on_device)
{
    return rows_copy(s, level, row0, nrows, dst, dst_on_device, true);
}

int ps_set_rows(ps_solver* s, int level, int row0, int nrows, const double* src, int src_on_device)
{
    if (s && !s->have_state) return fail(s, PS_ERR_STATE, "ps_set_rows before ps_set_state");
    return rows_copy(s, level, row0, nrows, const_cast<double*>(src), src_on_device, false);
}

int ps_synchronize(ps_solver* s)
{
    if (!s) return PS_ERR_INVALID;
    PS_CUDA(s, cudaSetDevice(s->device));
    PS_CUDA(s, cudaStreamSynchronize(s->stream));
    return drain_profile(s);
}

int ps_profile(ps_solver* s, int enable)
{
    if (!s) return PS_ERR_INVALID;
    int rc = ps_synchronize(s);
    if (rc) return rc;
    s->profile = enable != 0;
    for (int i = 0; i < 8; ++i) {
        s->prof_ms[i] = 0;
        s->prof_n[i] = 0;
        s->prof_cells[i] = 0;
    }
    return PS_OK;
}

int ps_profile_read(ps_solver* s, int kind, double* ms, int64_t* launches, double* cells)
{
    if (!s || kind < 0 || kind >= 8) return PS_ERR_INVALID;
    int rc = ps_synchronize(s);
    if (rc) return rc;
    if (ms) *ms = s->prof_ms[kind];
    if (launches) *launches = s->prof_n[kind];
    if (cells) *cells = s->prof_cells[kind];
    return PS_OK;
}

int ps_set_stream(ps_solver* s, void* stream)
{
    if (!s) return PS_ERR_INVALID;
    if (s->own_stream && s->stream) {
        cudaStreamSynchronize(s->stream);
        cudaStreamDestroy(s->stream);
    }
    if (stream) {
        s->stream = (cudaStream_t)stream;
        s->own_stream = false;
    } else {
        PS_CUDA(s, cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
        s->own_stream = true;
    }
    return PS_OK;
}

}  // extern "C"

// ====================================================================== batch
// Many independent instances in one set of launches (include/pysweep_b200.h,
// ps_batch_*).

struct BatchInst {
    int nx = 0, ny = 0, nb = 0, nseg = 1;
    double* base[2] = {nullptr, nullptr};
    double* xface = nullptr;
    double* yface = nullptr;
    size_t yface_n = 0;  // elements of both y-face buffers
    bool have_state = false;
    // levels advanced since this instance's state was set: the step function
    // of the next level sees globalTimeStep = level + 1, as one solver run of
    // all levels so far would show it (the reference starts at 1,
    // pysweep/core/solver.py:162)
    int64_t level = 0;
    std::map<std::string, double> globals;
};

struct ps_batch {
    int device = 0, eq = 0, nv = 1, ops = 1, its = 1, bs = 0, mpss = 0, H = 0;
    int chunk = 32;  // column chunk of the generic streams (32 or 64)
    bool fast = false;
    cudaStream_t stream = nullptr;
    // the gap stream runs beside the y-bridge on a high-priority side stream
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    std::vector<BatchInst> inst;
    SweptArgs* d_desc = nullptr;  // [count][2 roles][2 parities] (batch.cuh)
    int2* d_units = nullptr;      // (instance, unit) of every band segment
    int nunits = 0;
    int cur = 0;                  // base holding the current levels (all instances)
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    int64_t graph_levels = -1;
    int graph_cur = -1;
    int64_t graph_launches = 0;
    int64_t launches = 0;
    // the instances' level counters the device descriptors were uploaded with
    std::vector<int64_t> desc_level;
    // heat in overlapped blocks: the instances, and one table of (instance,
    // unit) pairs per block size in use
    BlockInst* d_binst = nullptr;
    bool binst_current = false;
    // Euler level by level: the instances with their level counters
    MarchInst* d_minst = nullptr;
    struct Table {
        int vw, vh, n;
        int2* d;
    };
    std::vector<Table> tables;
    std::string err;
};

namespace {

int bfail(ps_batch* b, int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (b) b->err = buf;
    else g_create_error = buf;
    return code;
}

#define PSB_CUDA(b, call)                                                                       \
    do {                                                                                        \
        cudaError_t e_ = (call);                                                                \
        if (e_ != cudaSuccess)                                                                  \
            return bfail((b), e_ == cudaErrorMemoryAllocation ? PS_ERR_NOMEM : PS_ERR_CUDA,     \
                         "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
    } while (0)

bool global_allowed(int eq, const char* name)
{
    for (const auto& g : kGlobals)
        if (!strcmp(g.name, name) && (g.eqmask >> eq & 1)) return true;
    return false;
}

void batch_free_graph(ps_batch* b)
{
    if (b->gexec) cudaGraphExecDestroy(b->gexec);
    if (b->graph) cudaGraphDestroy(b->graph);
    b->gexec = nullptr;
    b->graph = nullptr;
    b->graph_levels = -1;
}

// Upload both descriptors of every instance (constants may have changed).
int batch_upload(ps_batch* b)
{
    const int n = (int)b->inst.size();
    std::vector<SweptArgs> d(4 * n);
    const int O2 = 2 * b->ops;
    for (int i = 0; i < n; ++i) {
        const BatchInst& I = b->inst[i];
        for (int q = 0; q < 4; ++q) {
            const int role = q / 2, par = q % 2;
            SweptArgs& a = d[4 * i + q];
            memset(&a, 0, sizeof a);
            a.bin = I.base[par];
            a.bout = I.base[1 - par];
            a.xface = I.xface;
            a.yface = I.yface + (role ? I.yface_n / 2 : 0);
            a.frame_every = 1;
            a.nx = I.nx;
            a.ny = I.ny;
            a.nv = b->nv;
            a.bx = b->bs;
            a.hx = b->bs / 2;
            a.Hmax = b->H;
            a.nb = I.nb;
            a.nseg = I.nseg;
            a.wy = I.ny / I.nseg;
            a.nchunks = (a.wy + b->chunk - 1) / b->chunk;
            a.seg_unit = a.wy;
            a.seg_units = I.nseg;
            a.off = par ? b->bs / 2 : 0;  // prism bands alternate by half a block
            a.its = b->its;
            a.gts_base = (int)I.level;
            a.p = make_params_g(b->eq, I.globals);
            a.seam_direct = seam_direct(b->bs, b->ops, b->nv, b->its, b->H, sizeof(double)) ? 1 : 0;
        }
        (void)O2;
    }
    PSB_CUDA(b, cudaMemcpyAsync(b->d_desc, d.data(), d.size() * sizeof(SweptArgs),
                                cudaMemcpyHostToDevice, b->stream));
    PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    b->desc_level.resize(n);
    for (int i = 0; i < n; ++i) b->desc_level[i] = b->inst[i].level;
    return PS_OK;
}

// Whether the uploaded descriptors carry the instances' current level counters
// (the captured graph reads the descriptors from device memory at every replay).
bool batch_desc_current(const ps_batch* b)
{
    if (b->desc_level.size() != b->inst.size()) return false;
    for (size_t i = 0; i < b->inst.size(); ++i)
        if (b->desc_level[i] != b->inst[i].level) return false;
    return true;
}

size_t batch_tile_smem(const ps_batch* b)
{
    const int O2 = 2 * b->ops, RS = b->chunk + O2;
    return sizeof(double) * ((size_t)(b->its + 1) * b->nv * b->bs * RS +
                             (size_t)(b->H + 1) * b->nv * b->bs * O2);
}

size_t batch_stream_smem(const ps_batch* b)
{
    return batch_tile_smem(b);
}

size_t batch_seam_smem(const ps_batch* b)
{
    if (seam_direct(b->bs, b->ops, b->nv, b->its, b->H, sizeof(double)))
        return sizeof(double) * (size_t)(b->its + 1) * b->nv * b->bs * (2 * b->ops * (b->H + 1));
    return sizeof(double) * std::max(seam_smem_elems(false, b->bs, b->ops, b->nv, b->its, b->H),
                                     seam_smem_elems(true, b->bs, b->ops, b->nv, b->its, b->H));
}

// Enqueue one half-cycle for every instance: P, then Y on the batch stream
// beside G on the side stream (G reads nothing Y writes; see run_swept), then
// O after both.
template <class Eq, int ITS, int W>
void batch_half(ps_batch* b, int par, int H, long long L0, size_t ssm, size_t gsm)
{
    const int nu = b->nunits;
    cudaStream_t st = b->stream, sd = b->side;
    auto fork = [&] {
        cudaEventRecord(b->ev_fork, st);
        cudaStreamWaitEvent(sd, b->ev_fork, 0);
    };
    auto join = [&] {
        cudaEventRecord(b->ev_join, sd);
        cudaStreamWaitEvent(st, b->ev_join, 0);
    };
    stream_batch<Eq, ITS, W, false, 256><<<nu, 256, gsm, st>>>(b->d_desc, b->d_units, par, H, L0);
    fork();
    stream_batch<Eq, ITS, W, true, 256><<<nu, 256, gsm, sd>>>(b->d_desc, b->d_units, par, H, L0);
    seam_batch<Eq, ITS, false, 128><<<nu, 128, ssm, st>>>(b->d_desc, b->d_units, par, H, L0);
    join();
    seam_batch<Eq, ITS, true, 128><<<nu, 128, ssm, st>>>(b->d_desc, b->d_units, par, H, L0);
}

template <class Eq, int ITS, int W>
void batch_prepare()
{
    allow_big_smem(stream_batch<Eq, ITS, W, false, 256>);
    allow_big_smem(stream_batch<Eq, ITS, W, true, 256>);
    allow_big_smem(seam_batch<Eq, ITS, false, 128>);
    allow_big_smem(seam_batch<Eq, ITS, true, 128>);
}

using HalfFn = void (*)(ps_batch*, int, int, long long, size_t, size_t);
using PrepFn = void (*)();

bool batch_pick(int eq, int ops, int its, int chunk, HalfFn* half, PrepFn* prep)
{
#define PS_BSET(EQ, OP, IT, W, T)                                   \
    if (eq == EQ && ops == OP && its == IT && chunk == W) {         \
        *half = batch_half<T, IT, W>;                               \
        *prep = batch_prepare<T, IT, W>;                            \
        return true;                                                \
    }
    PS_BSET(PS_EQ_HEAT, 1, 1, 32, Heat)
    PS_BSET(PS_EQ_HEAT, 1, 2, 32, Heat)
    PS_BSET(PS_EQ_HALF, 1, 2, 32, Half)
#undef PS_BSET
    *half = nullptr;  // Euler runs level by level
    *prep = nullptr;
    return eq == PS_EQ_EULER && ops == 2 && its == 2;
}

// ---- heat in overlapped blocks (b->fast) ----
struct BlockStep {
    bool stream;
    TileShape tile;
    int T, table;
};

// The table of a block size, built on first use.  (Block sizes come from the
// tile shapes and level counts, so a batch has a few hundred at most.)
int batch_table(ps_batch* b, int vw, int vh, int* index)
{
    for (size_t i = 0; i < b->tables.size(); ++i)
        if (b->tables[i].vw == vw && b->tables[i].vh == vh) {
            *index = (int)i;
            return PS_OK;
        }
    std::vector<int2> u;
    for (int i = 0; i < (int)b->inst.size(); ++i) {
        const BatchInst& I = b->inst[i];
        const int n = ((I.ny + vw - 1) / vw) * ((I.nx + vh - 1) / vh);
        for (int k = 0; k < n; ++k) u.push_back(make_int2(i, k));
    }
    int2* d = nullptr;
    PSB_CUDA(b, cudaMalloc(&d, u.size() * sizeof(int2)));
    // (on the batch's own stream: it does not wait for the legacy one, and a copy
    // from pageable memory may return before it lands)
    cudaError_t e = cudaMemcpyAsync(d, u.data(), u.size() * sizeof(int2), cudaMemcpyHostToDevice, b->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
    if (e != cudaSuccess) {
        cudaFree(d);
        return bfail(b, PS_ERR_CUDA, "block table: %s", cudaGetErrorString(e));
    }
    b->tables.push_back({vw, vh, (int)u.size(), d});
    *index = (int)b->tables.size() - 1;
    return PS_OK;
}

// The launches of a run of nlevels levels, with their tables.
int batch_block_steps(ps_batch* b, int64_t nlevels, std::vector<BlockStep>* steps)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    std::vector<BlockGrid> gs;
    for (const auto& I : b->inst) gs.push_back({I.nx, I.ny});
    const BlockGrids g{gs.data(), (int)gs.size()};
    if (nlevels <= 0) return PS_OK;
    const BlockPlan plan = plan_block(kTilesFE, g, (int)std::min<int64_t>(nlevels, 1 << 20), 1,
                                      kTileMaxT, sms);
    const int rows = stream_rows(g, sms);
    BlockStep s{};
    int T = 0;
    for (int64_t done = 0; done < nlevels; done += T) {
        const int t = plan_next(plan, nlevels - done, 1);
        if (t != T) {
            T = t;
            s.T = T;
            s.stream = plan.stream && T == kStreamT;
            double us;
            if (!s.stream) s.tile = best_tile(kTilesFE, T, g, sms, &us);
            const int vw = s.stream ? kStreamW : tile_vw(s.tile, T);
            const int vh = s.stream ? rows : tile_vh(s.tile, T);
            if (int rc = batch_table(b, vw, vh, &s.table)) return rc;
        }
        steps->push_back(s);
    }
    return PS_OK;
}

int batch_block_upload(ps_batch* b)
{
    if (b->binst_current) return PS_OK;
    std::vector<BlockInst> d;
    for (const auto& I : b->inst)
        d.push_back({{I.base[0], I.base[1]}, make_params_g(b->eq, I.globals).d[0], I.nx, I.ny});
    PSB_CUDA(b, cudaMemcpyAsync(b->d_binst, d.data(), d.size() * sizeof(BlockInst),
                                cudaMemcpyHostToDevice, b->stream));
    PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    b->binst_current = true;
    return PS_OK;
}

template <int C, int R, int MAXW>
void launch_tile_batch(ps_batch* b, const BlockStep& s, const ps_batch::Table& t, int par)
{
    auto k = heat_block_tile_batch<C, R, MAXW>;
    const size_t smem = tile_smem<C>(s.tile.nw);
    if (smem > 48 * 1024) allow_big_smem(k);
    launch_after(k, t.n, 32 * s.tile.nw, smem, b->stream, (const BlockInst*)b->d_binst,
                 (const int2*)t.d, par, s.T, t.vw, t.vh);
}

int batch_block_enqueue(ps_batch* b, const std::vector<BlockStep>& steps)
{
    int par = b->cur;
    for (const BlockStep& s : steps) {
        const ps_batch::Table& t = b->tables[s.table];
        if (s.stream)
            launch_after(heat_block_stream_batch<double>, t.n, 32, 0, b->stream, (const BlockInst*)b->d_binst,
                         (const int2*)t.d, par, t.vh);
        else if (s.tile.R == 10) launch_tile_batch<4, 10, 12>(b, s, t, par);
        else if (s.tile.C == 4 && s.tile.R == 8) launch_tile_batch<4, 8, 16>(b, s, t, par);
        else if (s.tile.C == 4) launch_tile_batch<4, 6, 16>(b, s, t, par);
        else if (s.tile.R == 8) launch_tile_batch<2, 8, 20>(b, s, t, par);
        else launch_tile_batch<2, 4, 24>(b, s, t, par);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return bfail(b, PS_ERR_CUDA, "batched launch: %s", cudaGetErrorString(e));
        par ^= 1;
    }
    return PS_OK;
}

// ---- Euler level by level ----
int batch_march_upload(ps_batch* b)
{
    std::vector<MarchInst> d;
    for (const auto& I : b->inst) {
        const EqParams p = make_params_g(b->eq, I.globals);
        d.push_back({{I.base[0], I.base[1]}, p.d[0], p.d[1], p.d[2], p.d[3], I.nx, I.ny, (int)I.level});
    }
    PSB_CUDA(b, cudaMemcpyAsync(b->d_minst, d.data(), d.size() * sizeof(MarchInst),
                                cudaMemcpyHostToDevice, b->stream));
    PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    b->desc_level.clear();
    for (const auto& I : b->inst) b->desc_level.push_back(I.level);
    return PS_OK;
}

// Rows of the strips, and their table.
int batch_march_plan(ps_batch* b, int* hs, int* table)
{
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    std::vector<BlockGrid> gs;
    for (const auto& I : b->inst) gs.push_back({I.nx, I.ny});
    *hs = march_rows(BlockGrids{gs.data(), (int)gs.size()}, sms);
    return batch_table(b, kMarchW, *hs, table);
}

int batch_march_enqueue(ps_batch* b, int64_t nlevels, int hs, int table)
{
    const ps_batch::Table& t = b->tables[table];
    bool safe = true;  // (one kernel for all instances)
    for (const auto& I : b->inst) safe = safe && march_constants(make_params_g(b->eq, I.globals));
    const auto kernel = safe ? euler_march_batch<false> : euler_march_batch<true>;
    int older = 2 * b->cur, newest = older + 1;  // as in run_levels
    for (int64_t L = 1; L <= nlevels; ++L) {
        const int next = (newest + 1) % 4;
        launch_after(kernel, t.n, 32, 0, b->stream, (const MarchInst*)b->d_minst,
                     (const int2*)t.d, newest, older, next, hs, (int)L);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return bfail(b, PS_ERR_CUDA, "batched launch: %s", cudaGetErrorString(e));
        older = newest;
        newest = next;
    }
    if (newest % 2 == 0)
        for (auto& I : b->inst) {
            const size_t fe = (size_t)4 * I.nx * I.ny;
            auto slot = [&](int q) { return I.base[q / 2] + (size_t)(q % 2) * fe; };
            PSB_CUDA(b, cudaMemcpyAsync(slot(newest + 1), slot(newest), fe * sizeof(double),
                                        cudaMemcpyDeviceToDevice, b->stream));
            PSB_CUDA(b, cudaMemcpyAsync(slot(newest), slot(older), fe * sizeof(double),
                                        cudaMemcpyDeviceToDevice, b->stream));
        }
    return PS_OK;
}

// Enqueue a whole run of nlevels levels, starting from parity b->cur.
int batch_enqueue(ps_batch* b, int64_t nlevels, HalfFn half, int64_t* nlaunch)
{
    const size_t ssm = batch_seam_smem(b), gsm = batch_stream_smem(b);
    const size_t fe = (size_t)b->nv;
    int par = b->cur;
    int64_t done = 0, n = 0;
    while (done < nlevels) {
        const int H = (int)std::min<int64_t>(b->H, nlevels - done);
        if (H < b->its) {  // the newest its-H base levels carry over unchanged
            for (auto& I : b->inst) {
                const size_t f = fe * I.nx * I.ny;
                for (int q = 0; q < b->its - H; ++q)
                    PSB_CUDA(b, cudaMemcpyAsync(I.base[1 - par] + (size_t)q * f,
                                                I.base[par] + (size_t)(q + H) * f, f * sizeof(double),
                                                cudaMemcpyDeviceToDevice, b->stream));
            }
        }
        half(b, par, H, done, ssm, gsm);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return bfail(b, PS_ERR_CUDA, "batched launch: %s", cudaGetErrorString(e));
        n += 4;
        par ^= 1;
        done += H;
    }
    *nlaunch = n;
    return PS_OK;
}

}  // namespace

extern "C" {

int ps_batch_destroy(ps_batch* b);

int ps_batch_create(ps_batch** out, int device, int equation, int count, const int* nx,
                    const int* ny, int nv, int ops, int its, int blocksize)
{
    if (!out || count <= 0 || !nx || !ny) return bfail(nullptr, PS_ERR_INVALID, "bad arguments");
    *out = nullptr;
    HalfFn half;
    PrepFn prep;
    if (!batch_pick(equation, ops, its, 32, &half, &prep))
        return bfail(nullptr, PS_ERR_UNSUPPORTED, "no batched kernels for equation %d ops %d its %d",
                     equation, ops, its);
    if (equation == PS_EQ_EULER && nv != 4) return bfail(nullptr, PS_ERR_INVALID, "euler needs nv=4");
    if ((equation == PS_EQ_HEAT || equation == PS_EQ_HALF) && nv != 1)
        return bfail(nullptr, PS_ERR_INVALID, "heat/half need nv=1");
    if (blocksize % (2 * ops) || blocksize / (2 * ops) - 1 < 1)
        return bfail(nullptr, PS_ERR_INVALID, "blocksize %d invalid for ops %d", blocksize, ops);
    ps_batch* b = new ps_batch();
    b->device = device;
    b->eq = equation;
    b->nv = nv;
    b->ops = ops;
    b->its = its;
    b->bs = blocksize;
    b->mpss = blocksize / (2 * ops) - 1;
    b->H = default_levels(equation, its, blocksize, b->mpss);
    b->fast = equation == PS_EQ_HEAT && its == 1 && (blocksize == 16 || blocksize == 32);
    int rc = PS_OK;
    std::vector<int2> units;
    for (int i = 0; i < count && rc == PS_OK; ++i) {
        BatchInst I;
        I.nx = nx[i];
        I.ny = ny[i];
        if (I.nx % blocksize || I.ny % blocksize || (b->fast && I.ny % 32))
            rc = bfail(b, PS_ERR_INVALID, "instance %d: %dx%d not divisible by blocksize %d%s", i,
                       I.nx, I.ny, blocksize, b->fast ? " and 32" : "");
        else if ((size_t)3 * nv * I.nx * I.ny >= (size_t)1 << 31)
            rc = bfail(b, PS_ERR_UNSUPPORTED, "instance %d too large for 32-bit offsets", i);
        else if (!b->fast && 32 < 2 * ops * (b->H + 1))
            rc = bfail(b, PS_ERR_UNSUPPORTED, "blocksize %d too large for the batched streams", blocksize);
        I.nb = I.nx / blocksize;
        // heat in blocks needs no segments (the count is only reported); the
        // prisms: segments of about 256 columns that divide ny and hold a
        // chunk, so that the units of large and small instances take similar
        // times (a phase waits for its slowest unit)
        if (b->fast) {
            I.nseg = std::max(1, I.ny / 512);
        } else {
            const int minw = std::max(b->chunk, 2 * ops * (b->H + 1));
            I.nseg = 1;
            for (int q = 2; q <= I.ny / 256 && I.ny / q >= minw; ++q)
                if (I.ny % q == 0) I.nseg = q;
        }
        for (int u = 0; u < I.nb * I.nseg; ++u) units.push_back(make_int2(i, u));
        b->inst.push_back(I);
    }
    if (rc == PS_OK && batch_seam_smem(b) > 227 * 1024)
        rc = bfail(b, PS_ERR_UNSUPPORTED, "seam tile needs %zu bytes of shared memory",
                   batch_seam_smem(b));
    if (rc == PS_OK) {
        cudaError_t e = cudaSetDevice(device);
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
        int lo = 0, hi = 0;
        if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&lo, &hi);
        if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&b->side, cudaStreamNonBlocking, hi);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_join, cudaEventDisableTiming);
        if (e != cudaSuccess) rc = bfail(b, PS_ERR_CUDA, "stream: %s", cudaGetErrorString(e));
    }
    const int O2 = 2 * ops, HF = b->H - 1;
    for (auto& I : b->inst) {
        if (rc != PS_OK) break;
        const size_t f = (size_t)nv * I.nx * I.ny;
        const size_t xn = (size_t)I.nb * HF * 2 * nv * O2 * I.ny;
        // two y-face buffers: prism -> y-bridge and gap -> octahedron
        const size_t yn = 2 * (size_t)I.nb * I.nseg * 2 * HF * nv * blocksize * O2;
        I.yface_n = yn;
        cudaError_t e = cudaMalloc(&I.base[0], f * its * sizeof(double));
        if (e == cudaSuccess) e = cudaMalloc(&I.base[1], f * its * sizeof(double));
        // (blocks and single levels keep no faces)
        const bool faces = !b->fast && equation != PS_EQ_EULER;
        if (e == cudaSuccess && xn && faces) e = cudaMalloc(&I.xface, xn * sizeof(double));
        if (e == cudaSuccess && yn && faces) e = cudaMalloc(&I.yface, yn * sizeof(double));
        if (e != cudaSuccess) rc = bfail(b, PS_ERR_NOMEM, "instance buffers: %s", cudaGetErrorString(e));
    }
    if (rc == PS_OK) {
        b->nunits = (int)units.size();
        cudaError_t e = cudaMalloc(&b->d_desc, 4 * b->inst.size() * sizeof(SweptArgs));
        if (e == cudaSuccess && b->fast)
            e = cudaMalloc(&b->d_binst, b->inst.size() * sizeof(BlockInst));
        if (e == cudaSuccess && equation == PS_EQ_EULER)
            e = cudaMalloc(&b->d_minst, b->inst.size() * sizeof(MarchInst));
        if (e == cudaSuccess) e = cudaMalloc(&b->d_units, units.size() * sizeof(int2));
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(b->d_units, units.data(), units.size() * sizeof(int2),
                                cudaMemcpyHostToDevice, b->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(b->stream);
        if (e != cudaSuccess) rc = bfail(b, PS_ERR_NOMEM, "batch tables: %s", cudaGetErrorString(e));
    }
    // the kernels of the chosen chunk width (prep opts them into large shared memory)
    if (rc == PS_OK && !batch_pick(equation, ops, its, b->chunk, &half, &prep))
        rc = bfail(b, PS_ERR_UNSUPPORTED, "no batched kernels for chunk %d", b->chunk);
    if (rc == PS_OK && prep) prep();
    if (rc != PS_OK) {
        g_create_error = b->err;
        ps_batch_destroy(b);
        return rc;
    }
    *out = b;
    return PS_OK;
}

int ps_batch_destroy(ps_batch* b)
{
    if (!b) return PS_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    batch_free_graph(b);
    for (auto& I : b->inst) {
        for (auto& p : I.base)
            if (p) cudaFree(p);
        if (I.xface) cudaFree(I.xface);
        if (I.yface) cudaFree(I.yface);
    }
    if (b->d_binst) cudaFree(b->d_binst);
    if (b->d_minst) cudaFree(b->d_minst);
    for (auto& t : b->tables) cudaFree(t.d);
    if (b->d_desc) cudaFree(b->d_desc);
    if (b->d_units) cudaFree(b->d_units);
    if (b->side) {
        cudaStreamSynchronize(b->side);
        cudaStreamDestroy(b->side);
    }
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    if (b->ev_join) cudaEventDestroy(b->ev_join);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return PS_OK;
}

int ps_batch_set_global(ps_batch* b, int index, const char* name, const void* value, size_t nbytes)
{
    if (!b || !name || !value) return PS_ERR_INVALID;
    if (!global_allowed(b->eq, name)) return bfail(b, PS_ERR_INVALID, "no constant named %s", name);
    if (nbytes != 1 && nbytes != 2 && nbytes != 4 && nbytes != 8)
        return bfail(b, PS_ERR_INVALID, "constant %s: unsupported size %zu", name, nbytes);
    if (index < -1 || index >= (int)b->inst.size()) return bfail(b, PS_ERR_INVALID, "index %d", index);
    const double v = decode_value(value, nbytes);
    for (int i = 0; i < (int)b->inst.size(); ++i)
        if (index == -1 || index == i) b->inst[i].globals[name] = v;
    batch_free_graph(b);  // constants live in the captured descriptors
    b->binst_current = false;
    return PS_OK;
}

int ps_batch_set_state(ps_batch* b, int index, const double* src, int levels, int src_on_device)
{
    if (!b || !src || index < 0 || index >= (int)b->inst.size()) return PS_ERR_INVALID;
    if (levels != 1 && levels != b->its) return bfail(b, PS_ERR_INVALID, "levels must be 1 or its");
    PSB_CUDA(b, cudaSetDevice(b->device));
    BatchInst& I = b->inst[index];
    const size_t f = (size_t)b->nv * I.nx * I.ny;
    for (int q = 0; q < b->its; ++q)
        PSB_CUDA(b, cudaMemcpyAsync(I.base[b->cur] + (size_t)q * f, src + (size_t)(levels == 1 ? 0 : q) * f,
                                    f * sizeof(double),
                                    src_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                                    b->stream));
    if (!src_on_device) PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    I.have_state = true;
    I.level = 0;
    return PS_OK;
}

int ps_batch_run(ps_batch* b, int64_t nlevels, int use_graph)
{
    if (!b) return PS_ERR_INVALID;
    if (nlevels < 0) return bfail(b, PS_ERR_INVALID, "negative level count");
    for (size_t i = 0; i < b->inst.size(); ++i)
        if (!b->inst[i].have_state) return bfail(b, PS_ERR_STATE, "instance %zu has no state", i);
    PSB_CUDA(b, cudaSetDevice(b->device));
    HalfFn half;
    PrepFn prep;
    batch_pick(b->eq, b->ops, b->its, b->chunk, &half, &prep);
    int64_t nsteps = (nlevels + b->H - 1) / b->H;  // half-cycles, or block launches
    std::vector<BlockStep> steps;
    const bool rebuild = !use_graph || !b->gexec || b->graph_levels != nlevels || b->graph_cur != b->cur;
    if (b->fast && rebuild) {
        int rc = batch_block_steps(b, nlevels, &steps);
        if (rc) return rc;
        nsteps = (int64_t)steps.size();
    } else if (b->fast) {
        nsteps = b->graph_launches;
    }
    // Euler: base buffers of two levels each, one launch per level
    const bool march = b->eq == PS_EQ_EULER;
    int hs = 0, table = 0;
    if (march) {
        nsteps = (nlevels + 1) / 2;  // (the newest level's base buffer changes every other level)
        if (int rc = batch_march_plan(b, &hs, &table)) return rc;
    }
    auto upload = [&]() -> int {
        return b->fast ? batch_block_upload(b) : (march ? batch_march_upload(b) : batch_upload(b));
    };
    auto enqueue = [&](int64_t* n) -> int {
        if (march) {
            *n = nlevels;
            return batch_march_enqueue(b, nlevels, hs, table);
        }
        if (!b->fast) return batch_enqueue(b, nlevels, half, n);
        *n = (int64_t)steps.size();
        return batch_block_enqueue(b, steps);
    };
    if (!use_graph) {
        int rc = upload();
        if (rc) return rc;
        int64_t n = 0;
        rc = enqueue(&n);
        if (rc) return rc;
        b->launches += n;
    } else {
        if (rebuild) {
            batch_free_graph(b);
            int rc = upload();
            if (rc) return rc;
            PSB_CUDA(b, cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
            int64_t n = 0;
            rc = enqueue(&n);
            cudaGraph_t g = nullptr;
            cudaError_t e = cudaStreamEndCapture(b->stream, &g);
            if (rc) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            if (e != cudaSuccess) return bfail(b, PS_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
            b->graph = g;
            PSB_CUDA(b, cudaGraphInstantiate(&b->gexec, g, 0));
            b->graph_levels = nlevels;
            b->graph_cur = b->cur;
            b->graph_launches = n;
        } else if (!b->fast && !batch_desc_current(b)) {
            int rc = upload();  // new level counters for the same graph
            if (rc) return rc;
        }
        PSB_CUDA(b, cudaGraphLaunch(b->gexec, b->stream));
        b->launches += b->graph_launches;
    }
    b->cur ^= (int)(nsteps & 1);
    for (auto& I : b->inst) I.level += nlevels;
    return PS_OK;
}

int ps_batch_get_state(ps_batch* b, int index, double* dst, int level, int dst_on_device)
{
    if (!b || !dst || index < 0 || index >= (int)b->inst.size()) return PS_ERR_INVALID;
    if (level < 0 || level >= b->its) return bfail(b, PS_ERR_INVALID, "level %d", level);
    PSB_CUDA(b, cudaSetDevice(b->device));
    BatchInst& I = b->inst[index];
    const size_t f = (size_t)b->nv * I.nx * I.ny;
    if (!dst_on_device) map_host_pages(dst, f * sizeof(double));
    PSB_CUDA(b, cudaMemcpyAsync(dst, I.base[b->cur] + (size_t)(b->its - 1 - level) * f,
                                f * sizeof(double),
                                dst_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost,
                                b->stream));
    if (!dst_on_device) PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    return PS_OK;
}

int ps_batch_synchronize(ps_batch* b)
{
    if (!b) return PS_ERR_INVALID;
    PSB_CUDA(b, cudaSetDevice(b->device));
    PSB_CUDA(b, cudaStreamSynchronize(b->stream));
    return PS_OK;
}

int64_t ps_batch_launches(const ps_batch* b) { return b ? b->launches : 0; }

const char* ps_batch_last_error(const ps_batch* b) { return b ? b->err.c_str() : g_create_error.c_str(); }

int ps_batch_units(const ps_batch* b) { return b ? b->nunits : 0; }

}  // extern "C"
