// ps_heat_swept_noalloc: the swept heat path for callers that cannot allocate
// device memory.
//
// Some hosts of this library run where a cudaMalloc is not allowed at call
// time: plugins of a process whose memory pool owns the whole device, or
// real-time loops that must not touch the allocator.  This entry point takes
// only the caller's input and output fields and keeps every temporary buffer
// in one file-scope device array, g_noalloc_scratch, that the CUDA runtime
// reserves on each device when the library is loaded.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "../../include/pysweep_b200.h"
#include "heat_block.cuh"

namespace {

// Scratch for one call: an intermediate field plus the prism faces.  Held by
// every GPU that loads the library, for the life of the process.
constexpr size_t kScratchBytes = (size_t)128 << 20;  // 128 MiB
__device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_mu;
void* g_scratch_ptr[kMaxDevices] = {};

void put_err(char* err, size_t errlen, const char* msg)
{
    if (err && errlen) {
        strncpy(err, msg, errlen - 1);
        err[errlen - 1] = '\0';
    }
}

size_t round_up(size_t v) { return (v + 255) & ~(size_t)255; }

// Whether the byte ranges [a, a+na) and [b, b+nb) share a byte.
bool overlap(const void* a, size_t na, const void* b, size_t nb)
{
    const uintptr_t x = (uintptr_t)a, y = (uintptr_t)b;
    return x < y + nb && y < x + na;
}

}  // namespace

using namespace psb;

extern "C" int ps_heat_swept_noalloc(const double* d_in, double* d_out, int nx, int ny,
                                     int blocksize, int64_t nsteps, double alpha, double dt,
                                     double dx, void* stream, char* err, size_t errlen)
{
    char msg[256];
    if (!d_in || !d_out) {
        put_err(err, errlen, "d_in and d_out must be device pointers");
        return PS_ERR_INVALID;
    }
    if ((blocksize != 16 && blocksize != 32) || nx <= 0 || ny <= 0 || nx % blocksize ||
        ny % 64 || nsteps < 0) {
        snprintf(msg, sizeof msg,
                 "need blocksize 16 or 32, nx a multiple of it, ny a multiple of %d, nsteps >= 0 "
                 "(got bs %d, %dx%d, %lld steps)",
                 64, blocksize, nx, ny, (long long)nsteps);
        put_err(err, errlen, msg);
        return PS_ERR_INVALID;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const size_t fe = (size_t)nx * ny;
    int dev = 0;
    cudaGetDevice(&dev);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // the sizes this entry point has always taken: a field and the faces of a
    // prism decomposition in the scratch array (blocks need the field only)
    const int BX = blocksize, HF = BX / 2 - 2, nb = nx / BX;
    const int nseg = std::max(1, std::min(ny / 64, sms * (BX == 16 ? 16 : 12) / nb));
    const size_t field_b = round_up(fe * sizeof(double));
    const size_t xface_b = round_up((size_t)nb * HF * 2 * 2 * ny * sizeof(double));
    const size_t yface_b = round_up((size_t)nb * nseg * 2 * HF * BX * 2 * sizeof(double));
    const size_t need = field_b + xface_b + yface_b;
    if (need > kScratchBytes) {
        snprintf(msg, sizeof msg,
                 "%dx%d with blocksize %d needs %zu bytes of scratch; the built-in scratch "
                 "holds %zu bytes",
                 nx, ny, blocksize, need, kScratchBytes);
        put_err(err, errlen, msg);
        return PS_ERR_INVALID;
    }
    if (overlap(d_in, fe * sizeof(double), d_out, fe * sizeof(double))) {
        put_err(err, errlen, "d_in and d_out overlap: the solve reads d_in while it writes d_out");
        return PS_ERR_INVALID;
    }
    if (nsteps == 0) {
        cudaError_t e = cudaMemcpyAsync(d_out, d_in, fe * sizeof(double),
                                        cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) {
            put_err(err, errlen, cudaGetErrorString(e));
            return PS_ERR_CUDA;
        }
        return PS_OK;
    }
    if (dev < 0 || dev >= kMaxDevices) {
        put_err(err, errlen, "device ordinal out of range");
        return PS_ERR_INVALID;
    }
    // set-up, once per device: the device address of the scratch array (the
    // host-side symbol is not a device address)
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_mu);
        if (!g_scratch_ptr[dev]) {
            void* p = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess || !p) {
                snprintf(msg, sizeof msg, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
                put_err(err, errlen, msg);
                return PS_ERR_CUDA;
            }
            g_scratch_ptr[dev] = p;
        }
        base = g_scratch_ptr[dev];
    }
    if (overlap(d_in, fe * sizeof(double), base, need) ||
        overlap(d_out, fe * sizeof(double), base, need)) {
        put_err(err, errlen, "d_in or d_out lies inside the library's scratch array");
        return PS_ERR_INVALID;
    }
    // Overlapped blocks (heat_block.cuh), the launches and kernels of ps_run.
    // Outputs alternate between d_out and the scratch field so that the last
    // launch lands in d_out and d_in is only read
    const BlockGrid grid{nx, ny};
    const BlockGrids grids{&grid, 1};
    const BlockPlan plan = plan_block(kTilesFE, grids, (int)std::min<int64_t>(nsteps, 1 << 20), 1,
                                      kTileMaxT, sms);
    int64_t count = 0;
    for (int64_t done = 0; done < nsteps; ++count) done += plan_next(plan, nsteps - done, 1);
    BlockArgs a;
    memset(&a, 0, sizeof a);
    a.nx = nx;
    a.ny = ny;
    a.v4 = (uintptr_t)d_in % 32 == 0 && (uintptr_t)d_out % 32 == 0;
    a.cr = alpha * dt / dx / dx;  // heat.py:37
    a.in = d_in;
    int64_t done = 0;
    for (int64_t k = 0; k < count; ++k) {
        const int T = plan_next(plan, nsteps - done, 1);
        a.out = (count - 1 - k) % 2 == 0 ? d_out : (double*)base;
        double us;
        if (plan.stream && T == kStreamT) launch_block_stream<double, false>(a, sms, st);
        else launch_block_tile<double, false>(best_tile(kTilesFE, T, grids, sms, &us), a, T, st);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            snprintf(msg, sizeof msg, "kernel launch: %s", cudaGetErrorString(e));
            put_err(err, errlen, msg);
            return PS_ERR_CUDA;
        }
        a.in = a.out;
        done += T;
    }
    return PS_OK;
}
