// Heat equation with a spatially varying diffusivity and its adjoint.
//
// Forward, per cell (the heat plugin's operation order, pysweep/equations/
// heat.py:60-64, with the courant number per cell):
//     C = alpha * dt / dx / dx
//     u' = (C*((u[x+1]-2u)+u[x-1]) + C*((u[y+1]-2u)+u[y-1])) + u
// i.e. u_{n+1} = u_n + C .* (L u_n) with L the periodic 5-point Laplacian
// (symmetric).  For J(u_N), with lambda_n = dJ/du_n:
//     lambda_n = lambda_{n+1} + L (C .* lambda_{n+1})
//     dJ/dC   += lambda_{n+1} .* (L u_n),        dJ/dalpha = dJ/dC * dt/dx/dx
// The forward stores u every `every` steps; the backward pass walks the
// segments from the last to the first, steps a segment's state forward from its
// checkpoint, keeping it every few levels in a work buffer, then runs the
// adjoint backward through the segment, those few levels per launch.
//
// The levels run in overlapped tiles, several per launch (heatvar_block.cuh):
// the forward steps, and the adjoint levels, whose tile recomputes the levels'
// Laplacians on chip.  ps_heatvar_recompute stores a segment's Laplacians for
// the adjoint solvers, which read them.  Every cell sees the one-step operations
// in their order, so the number of levels per launch changes no bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../include/pysweep_b200.h"
#include "heatvar_block.cuh"

namespace psb {
namespace {

__global__ void courant_kernel(const double* __restrict__ alpha, double* __restrict__ C, size_t n,
                               double dt, double dx)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        C[i] = alpha[i] * dt / dx / dx;
}

__global__ void scale_kernel(double* __restrict__ g, size_t n, double f)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        g[i] *= f;
}

int sm_count()
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

VarArgs var_args(const double* C, int nx, int ny)
{
    VarArgs a;
    memset(&a, 0, sizeof a);
    a.C = C;
    a.nx = nx;
    a.ny = ny;
    return a;
}

// Levels of each launch of a run of n levels.
template <int ROLE>
std::vector<int> launches(int64_t n, int nx, int ny, int sms)
{
    std::vector<int> t;
    if (n <= 0) return t;
    const BlockGrid grid{nx, ny};
    const BlockPlan plan =
        plan_var<ROLE>(BlockGrids{&grid, 1}, (int)std::min<int64_t>(n, 1 << 20), sms);
    for (int64_t done = 0; done < n; done += t.back()) t.push_back(plan_next(plan, n - done, 1));
    return t;
}

// The Laplacians of the levels u, .., of a segment of `length` steps from u0
// into lap[0 .. length-1].  The states between launches alternate between two
// scratch fields so that the last one but one lands in s0.
void recompute(const double* C, const double* u0, double* lap, int length, int nx, int ny,
               double* s0, double* s1, int sms, cudaStream_t st)
{
    const size_t n = (size_t)nx * ny;
    const std::vector<int> t = launches<VAR_RECOMPUTE>(length, nx, ny, sms);
    VarArgs a = var_args(C, nx, ny);
    a.step = (long long)n;
    a.in = u0;
    size_t j = 0;
    for (size_t k = 0; k < t.size(); ++k) {
        const size_t left = t.size() - 1 - k;
        a.out = left == 0 ? nullptr : (left % 2 ? s0 : s1);
        a.lap = lap + j * n;
        launch_var<VAR_RECOMPUTE>(a, t[k], sms, st);
        a.in = a.out;
        j += t[k];
    }
}

}  // namespace
}  // namespace psb

using namespace psb;

namespace {
int adj_check(int nx, int ny, char* err, size_t errlen)
{
    if (nx < 3 || ny < 64 || ny % 64) {
        if (err && errlen) snprintf(err, errlen, "need nx >= 3 and ny a multiple of 64 (got %dx%d)", nx, ny);
        return PS_ERR_INVALID;
    }
    return PS_OK;
}

int adj_cuda(cudaError_t e, char* err, size_t errlen)
{
    if (e == cudaSuccess) return PS_OK;
    if (err && errlen) snprintf(err, errlen, "%s", cudaGetErrorString(e));
    return PS_ERR_CUDA;
}
}  // namespace

extern "C" int ps_heatvar_courant(const double* d_alpha, double* d_courant, int nx, int ny,
                                  double dt, double dx, void* stream, char* err, size_t errlen)
{
    int rc = adj_check(nx, ny, err, errlen);
    if (rc) return rc;
    if (!d_alpha || !d_courant) {
        if (err && errlen) snprintf(err, errlen, "bad arguments");
        return PS_ERR_INVALID;
    }
    courant_kernel<<<1024, 256, 0, (cudaStream_t)stream>>>(d_alpha, d_courant, (size_t)nx * ny, dt,
                                                          dx);
    return adj_cuda(cudaGetLastError(), err, errlen);
}

extern "C" int ps_heatvar_recompute(const double* d_courant, const double* d_u0, double* d_lap,
                                    int length, int nx, int ny, double* d_work, void* stream,
                                    char* err, size_t errlen)
{
    int rc = adj_check(nx, ny, err, errlen);
    if (rc) return rc;
    if (!d_courant || !d_u0 || !d_lap || !d_work || length < 0) {
        if (err && errlen) snprintf(err, errlen, "bad arguments");
        return PS_ERR_INVALID;
    }
    const size_t n = (size_t)nx * ny;
    recompute(d_courant, d_u0, d_lap, length, nx, ny, d_work, d_work + n, sm_count(),
              (cudaStream_t)stream);
    return adj_cuda(cudaGetLastError(), err, errlen);
}

extern "C" int ps_heatvar_forward(const double* d_u0, const double* d_alpha, double* d_uT, int nx,
                                  int ny, int64_t nsteps, double dt, double dx, double* d_courant,
                                  double* d_work, double* d_checkpoints, int every, void* stream,
                                  char* err, size_t errlen)
{
    int rc = adj_check(nx, ny, err, errlen);
    if (rc) return rc;
    if (!d_u0 || !d_alpha || !d_uT || !d_courant || !d_work || nsteps < 0 || every < 1) {
        if (err && errlen) snprintf(err, errlen, "bad arguments");
        return PS_ERR_INVALID;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const size_t n = (size_t)nx * ny;
    courant_kernel<<<1024, 256, 0, st>>>(d_alpha, d_courant, n, dt, dx);
    if (d_checkpoints)
        if ((rc = adj_cuda(cudaMemcpyAsync(d_checkpoints, d_u0, n * sizeof(double),
                                           cudaMemcpyDeviceToDevice, st), err, errlen)))
            return rc;
    if (nsteps == 0)
        return adj_cuda(cudaMemcpyAsync(d_uT, d_u0, n * sizeof(double), cudaMemcpyDeviceToDevice, st),
                        err, errlen);
    // launches end at the checkpoints, which take the state where they are;
    // between them it alternates between d_work and d_uT, the last in d_uT
    const int sms = sm_count();
    struct Step {
        int T;
        double* ck;
    };
    std::vector<Step> steps;
    for (int64_t done = 0; done < nsteps;) {
        const int64_t len = d_checkpoints ? std::min<int64_t>(every, nsteps - done) : nsteps - done;
        for (int T : launches<VAR_FORWARD>(len, nx, ny, sms)) steps.push_back({T, nullptr});
        done += len;
        if (d_checkpoints && done < nsteps) steps.back().ck = d_checkpoints + (size_t)(done / every) * n;
    }
    auto out = [&](size_t k) {
        return steps[k].ck ? steps[k].ck : ((steps.size() - 1 - k) % 2 == 0 ? d_uT : d_work);
    };
    VarArgs a = var_args(d_courant, nx, ny);
    a.in = d_u0;
    if (d_u0 == d_uT && out(0) == d_uT) {
        // in place: tiles overlap, so no launch may write the field it reads
        if (d_checkpoints) {
            a.in = d_checkpoints;
        } else {
            if ((rc = adj_cuda(cudaMemcpyAsync(d_work, d_u0, n * sizeof(double), cudaMemcpyDeviceToDevice,
                                               st), err, errlen)))
                return rc;
            a.in = d_work;
        }
    }
    for (size_t k = 0; k < steps.size(); ++k) {
        a.out = out(k);
        launch_var<VAR_FORWARD>(a, steps[k].T, sms, st);
        a.in = a.out;
    }
    return adj_cuda(cudaGetLastError(), err, errlen);
}

extern "C" int ps_heatvar_adjoint(const double* d_courant, const double* d_checkpoints, int every,
                                  const double* d_lamT, double* d_lam0, double* d_galpha, int nx,
                                  int ny, int64_t nsteps, double dt, double dx, double* d_states,
                                  double* d_lamwork, void* stream, char* err, size_t errlen)
{
    int rc = adj_check(nx, ny, err, errlen);
    if (rc) return rc;
    if (!d_courant || !d_checkpoints || !d_lamT || !d_lam0 || !d_galpha || !d_states ||
        !d_lamwork || every < 1 || nsteps < 0) {
        if (err && errlen) snprintf(err, errlen, "bad arguments");
        return PS_ERR_INVALID;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const size_t n = (size_t)nx * ny;
    const int sms = sm_count();
    const int64_t nseg = (nsteps + every - 1) / every;
    auto length = [&](int64_t k) { return (int)(std::min<int64_t>((k + 1) * every, nsteps) - k * every); };
    const BlockGrid grid{nx, ny};
    auto cut = [&](int n) {  // levels of each launch of a segment of n
        std::vector<int> t;
        const BlockPlan plan = plan_back(BlockGrids{&grid, 1}, n, sms);
        for (int done = 0; done < n; done += t.back()) t.push_back(plan_next(plan, n - done, 1));
        return t;
    };
    // every segment but the last has `every` steps
    const std::vector<int> whole = cut((int)std::min<int64_t>(every, nsteps));
    const std::vector<int> tail = cut(nseg ? length(nseg - 1) : 0);
    const int64_t count = nseg ? (int64_t)tail.size() + (nseg - 1) * (int64_t)whole.size() : 0;
    if ((rc = adj_cuda(cudaMemsetAsync(d_galpha, 0, n * sizeof(double), st), err, errlen))) return rc;
    // lambda ping-pong between d_lam0 and d_lamwork, arranged so that lambda_0
    // lands in d_lam0
    double* lam = count % 2 == 0 ? d_lam0 : d_lamwork;
    if ((rc = adj_cuda(cudaMemcpyAsync(lam, d_lamT, n * sizeof(double), cudaMemcpyDeviceToDevice, st),
                       err, errlen)))
        return rc;
    BackArgs a;
    memset(&a, 0, sizeof a);
    a.C = d_courant;
    a.g = d_galpha;
    a.nx = nx;
    a.ny = ny;
    VarArgs f = var_args(d_courant, nx, ny);
    for (int64_t k = nseg - 1; k >= 0; --k) {
        const std::vector<int>& t = k == nseg - 1 ? tail : whole;
        const double* u0 = d_checkpoints + (size_t)k * n;
        // the state every launch but the first starts from: d_states[0], [1], ..
        f.in = u0;
        for (size_t j = 0; j + 1 < t.size(); ++j) {
            f.out = d_states + j * n;
            launch_var<VAR_FORWARD>(f, t[j], sms, st);
            f.in = f.out;
        }
        for (size_t j = t.size(); j-- > 0;) {
            a.u = j ? d_states + (j - 1) * n : u0;
            a.in = lam;
            lam = lam == d_lam0 ? d_lamwork : d_lam0;
            a.out = lam;
            launch_back(a, t[j], sms, st);
        }
    }
    scale_kernel<<<1024, 256, 0, st>>>(d_galpha, n, dt / dx / dx);
    return adj_cuda(cudaGetLastError(), err, errlen);
}
