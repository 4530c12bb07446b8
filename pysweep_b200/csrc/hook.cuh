// User step hooks: the plugin's __device__ step() compiled at run time.
//
// The reference builds its kernels from the plugin's .cu file when a Solver
// starts (pysweep/core/io.py:146-155: SourceModule(pysweep.cu with
// -DPYSWEEP_GPU_SOURCE=<file>)) and copies the framework and plugin constants
// into the module's __constant__ variables by name (io.py:169-184,
// pysweep/equations/heat.py:38-46).  This file does the same with NVRTC for
// sm_100a: the hook's source is wrapped in the program of hook_program(),
// whose kernels (hook_kernels.cuh) run it inside the swept phases and a tiled
// standard step; the module is loaded with the driver API into the current
// (primary) context; constants are found by name in the three kernel-kind
// namespaces.  NVRTC is opened with dlopen on first use and the driver-API
// calls are resolved through the runtime (cudaGetDriverEntryPoint), so the
// library loads (and every built-in equation runs) where NVRTC is absent, and
// loads without a driver at all on a machine with no GPU.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <dlfcn.h>

#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

namespace psb {

// kernel kinds, each with its own namespace, tile geometry and constants
enum HookNs { HOOK_STREAM = 0, HOOK_SEAM = 1, HOOK_STD = 2 };
constexpr const char* kHookNs[3] = {"psh_stream", "psh_seam", "psh_std"};
// framework constants of pysweep/core/pysweep.cu:12-20, in this order
enum HookFw { FW_VARS, FW_TIMES, FW_MPSS, FW_MOSS, FW_NV, FW_OPS, FW_ITS, FW_SX, FW_SY, FW_COUNT };
constexpr const char* kHookFw[FW_COUNT] = {"VARS", "TIMES", "MPSS", "MOSS", "NV",
                                           "OPS",  "ITS",   "SX",   "SY"};
// block tiles of the hook kernels (hook_kernels.cuh): columns of level 1, most
// threads, most levels per launch.
constexpr int kHookBlkW = 64, kHookBlkNT = 512, kHookBlkMaxT = 8;

// Rows of level 1 and levels of a block, threads of a launch of one level (of
// several: kHookBlkNT), or rows 0 where no tile fits.
// Slots of levels -1 .. T; the deepest block whose last level keeps two thirds of
// the first one's cells and whose tile leaves room for two CTAs per SM; one level
// where a second does not fit.  Several levels run 512 threads (a step's loads may
// not pass the store of the step before it, so warps have to cover its latency;
// heat at 1024², us per level with 256 / 512 / 1024: 5.2, 4.6, 6.6).
//
// One level: as many rows as leave enough warps on an SM, a warp to a row.  A
// stencil of nv variables and reach ops, us per level with 32 rows and 256 threads
// / 16 and 256 / 8 and 256 / 16 and 512 (-: too large):
//     512²  nv 1 ops 1  7.8 / 6.3 / 5.9 / 5.9   nv 3 ops 2    - /  13 /  15 /  12
//     2048² nv 1 ops 1   42 /  44 /  53 /  60   nv 3 ops 2    - / 167 / 143 / 136
//           nv 2 ops 1  105 /  76 /  78 /  86   nv 4 ops 1    - / 209 / 146 / 177
//           nv 4 ops 2    - /   - / 240 / 267   nv 6 ops 2    - /   - / 569 / 373
// so 32 rows where four CTAs fit on an SM and there are eight for each, 16 where
// three fit; else 16 with 512 threads where two do and the halo is wide (eight rows
// load half as much again), 8 where two do, 16 with 512 threads where one does.
struct HookBlock {
    int rows, T, threads1;
};
inline size_t hook_block_smem(int nv, int ops, int rows, int T)
{
    return sizeof(double) * (T + 2) * nv * (rows + 2 * ops) * (kHookBlkW + 2 * ops);
}
inline HookBlock hook_block(int nv, int ops, int maxT, long long cells, int sms)
{
    constexpr int few = kHookBlkNT / 2;
    for (int rows : {32, 16})
        for (int T = maxT < kHookBlkMaxT ? maxT : kHookBlkMaxT; T >= 2; --T) {
            const int ih = rows - 2 * ops * (T - 1), iw = kHookBlkW - 2 * ops * (T - 1);
            const size_t sm = hook_block_smem(nv, ops, rows, T);
            if (ih > 0 && iw > 0 && 3 * ih * iw >= 2 * rows * kHookBlkW && sm <= 113 * 1024)
                return HookBlock{rows, T, few};
        }
    auto fit = [&](int rows) {  // CTAs on an SM: 228 KB, 1 KB for each besides its own
        return (int)(228 * 1024 / (hook_block_smem(nv, ops, rows, 1) + 1024));
    };
    if (fit(32) >= 4 && cells >= 8LL * sms * 32 * kHookBlkW) return HookBlock{32, 1, few};
    if (fit(16) >= 3) return HookBlock{16, 1, few};
    if (fit(16) >= 2 && ops >= 2) return HookBlock{16, 1, kHookBlkNT};
    if (fit(8) >= 2) return HookBlock{8, 1, few};
    if (fit(16) >= 1) return HookBlock{16, 1, kHookBlkNT};
    for (int rows : {8, 4})
        if (fit(rows) >= 1) return HookBlock{rows, 1, few};
    return HookBlock{0, 0, 0};
}

// A user constant, in every namespace (ps_get_global hands out a pointer to
// it; `name` comes first, as in the built-in constants' table).
struct HookConst {
    const char* name = nullptr;
    size_t size = 0;
    CUdeviceptr ptr[3] = {0, 0, 0};
};

struct HookModule {
    CUmodule mod = nullptr;
    CUfunction prism[2] = {nullptr, nullptr};  // chunk 32, 64
    CUfunction gap[2] = {nullptr, nullptr};
    CUfunction ybridge = nullptr, octahedron = nullptr, block = nullptr;
    CUdeviceptr fw[3][FW_COUNT] = {};
    int fw_val[3][FW_COUNT];  // last values written (-1: never)
    std::map<std::string, HookConst> consts;
    int nv = 1, ops = 1, its = 1;
    HookModule()
    {
        for (auto& r : fw_val)
            for (int& v : r) v = -1;
    }
};

// ------------------------------------------------------------- driver API --
// The driver calls the hook path makes, resolved once from the driver the
// CUDA runtime loaded.
struct Driver {
    decltype(&cuModuleLoadData) moduleLoadData = nullptr;
    decltype(&cuModuleUnload) moduleUnload = nullptr;
    decltype(&cuModuleGetFunction) moduleGetFunction = nullptr;
    decltype(&cuModuleGetGlobal) moduleGetGlobal = nullptr;
    decltype(&cuFuncSetAttribute) funcSetAttribute = nullptr;
    decltype(&cuMemcpyHtoDAsync) memcpyHtoDAsync = nullptr;
    decltype(&cuLaunchKernel) launchKernel = nullptr;
    decltype(&cuLaunchKernelEx) launchKernelEx = nullptr;
    decltype(&cuGetErrorString) getErrorString = nullptr;
    bool ok = false;
};

inline Driver& drv()
{
    static Driver d;
    static std::once_flag once;
    std::call_once(once, [] {
        auto get = [](const char* sym, void** fn) {
            cudaDriverEntryPointQueryResult q;
            return cudaGetDriverEntryPoint(sym, fn, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess && *fn;
        };
        d.ok = get("cuModuleLoadData", (void**)&d.moduleLoadData) &&
               get("cuModuleUnload", (void**)&d.moduleUnload) &&
               get("cuModuleGetFunction", (void**)&d.moduleGetFunction) &&
               get("cuModuleGetGlobal", (void**)&d.moduleGetGlobal) &&
               get("cuFuncSetAttribute", (void**)&d.funcSetAttribute) &&
               get("cuMemcpyHtoDAsync", (void**)&d.memcpyHtoDAsync) &&
               get("cuLaunchKernel", (void**)&d.launchKernel) &&
               get("cuLaunchKernelEx", (void**)&d.launchKernelEx) &&
               get("cuGetErrorString", (void**)&d.getErrorString);
    });
    return d;
}

// ------------------------------------------------------------------ NVRTC --
// The handful of NVRTC entry points used, resolved from the shared library.
struct Nvrtc {
    using Create = int (*)(void**, const char*, const char*, int, const char* const*,
                           const char* const*);
    using Compile = int (*)(void*, int, const char* const*);
    using Size = int (*)(void*, size_t*);
    using Get = int (*)(void*, char*);
    using Destroy = int (*)(void**);
    Create create = nullptr;
    Compile compile = nullptr;
    Size log_size = nullptr, cubin_size = nullptr;
    Get log = nullptr, cubin = nullptr;
    Destroy destroy = nullptr;
    bool ok = false;
    std::string why;
};

inline Nvrtc& nvrtc()
{
    static Nvrtc n;
    static std::once_flag once;
    std::call_once(once, [] {
        const char* home = getenv("CUDA_HOME");
        std::vector<std::string> names = {"libnvrtc.so.12", "libnvrtc.so"};
        names.push_back(std::string(home ? home : "/usr/local/cuda") + "/lib64/libnvrtc.so.12");
        void* h = nullptr;
        for (const auto& nm : names)
            if ((h = dlopen(nm.c_str(), RTLD_NOW | RTLD_LOCAL))) break;
        if (!h) {
            n.why = "libnvrtc.so.12 not found (needed to compile step hooks)";
            return;
        }
        n.create = (Nvrtc::Create)dlsym(h, "nvrtcCreateProgram");
        n.compile = (Nvrtc::Compile)dlsym(h, "nvrtcCompileProgram");
        n.log_size = (Nvrtc::Size)dlsym(h, "nvrtcGetProgramLogSize");
        n.log = (Nvrtc::Get)dlsym(h, "nvrtcGetProgramLog");
        n.cubin_size = (Nvrtc::Size)dlsym(h, "nvrtcGetCUBINSize");
        n.cubin = (Nvrtc::Get)dlsym(h, "nvrtcGetCUBIN");
        n.destroy = (Nvrtc::Destroy)dlsym(h, "nvrtcDestroyProgram");
        n.ok = n.create && n.compile && n.log_size && n.log && n.cubin_size && n.cubin && n.destroy;
        if (!n.ok) n.why = "libnvrtc lacks an entry point";
    });
    return n;
}

// Directory of this library's kernel headers (csrc/ beside the .so).
inline std::string hook_include_dir()
{
    Dl_info info;
    if (dladdr((void*)&hook_include_dir, &info) && info.dli_fname) {
        std::string p = info.dli_fname;
        const size_t k = p.rfind('/');
        return (k == std::string::npos ? std::string(".") : p.substr(0, k)) + "/csrc";
    }
    return "csrc";
}

// The run-time program: the hook once per kernel kind, each copy in a
// namespace that declares the framework constants as the reference's
// pysweep.cu does (so the hook's VARS, TIMES, SY, ... resolve to them), then
// the kernels.
inline std::string hook_program(const std::string& src, const std::string& name, int nv, int ops,
                                int its)
{
    std::string p;
    p += "#define PSH_NV " + std::to_string(nv) + "\n";
    p += "#define PSH_OPS " + std::to_string(ops) + "\n";
    p += "#define PSH_ITS " + std::to_string(its) + "\n";
    p += "#define PSH_BLK_W " + std::to_string(kHookBlkW) + "\n";
    p += "#define PSH_BLK_NT " + std::to_string(kHookBlkNT) + "\n";
    p += "#define PSH_BLK_MAXT " + std::to_string(kHookBlkMaxT) + "\n";
    for (const char* ns : kHookNs) {
        p += std::string("namespace ") + ns + " {\n";
        p += "__device__ __constant__ int VARS, TIMES, MPSS, MOSS, NV, OPS, ITS, SX, SY;\n";
        p += "__device__ __constant__ const int LB_MIN_BLOCKS = 1;\n";
        p += "__device__ __constant__ const int LB_MAX_THREADS = 1024;\n";
        p += "#line 1 \"" + name + "\"\n";
        p += src;
        p += "\n}\n";
    }
    p += "#include \"hook_kernels.cuh\"\n";
    return p;
}

// Compile a program for sm_100a into a cubin; returns 0 or PS_ERR_* with the
// compiler's log in *log.  Cubins are cached per program text.
inline int hook_compile(const std::string& prog, std::vector<char>* cubin, std::string* log)
{
    static std::mutex mu;
    static std::map<std::string, std::vector<char>> cache;
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = cache.find(prog);
        if (it != cache.end()) {
            *cubin = it->second;
            return 0;
        }
    }
    Nvrtc& n = nvrtc();
    if (!n.ok) {
        *log = n.why;
        return -6;  // PS_ERR_COMPILE
    }
    void* h = nullptr;
    if (n.create(&h, prog.c_str(), "pysweep_hook.cu", 0, nullptr, nullptr) != 0) {
        *log = "nvrtcCreateProgram failed";
        return -6;
    }
    const std::string inc = "-I" + hook_include_dir();
    const char* opts[] = {"-arch=sm_100a", "--fmad=false", "-std=c++17", "-lineinfo",
                          "-diag-suppress=177,550", inc.c_str()};
    const int rc = n.compile(h, (int)(sizeof opts / sizeof *opts), opts);
    size_t ls = 0;
    n.log_size(h, &ls);
    std::string lg(ls, '\0');
    if (ls) n.log(h, &lg[0]);
    while (!lg.empty() && (lg.back() == '\0' || lg.back() == '\n')) lg.pop_back();
    *log = lg;
    if (rc != 0) {
        n.destroy(&h);
        return -6;
    }
    size_t cs = 0;
    n.cubin_size(h, &cs);
    cubin->assign(cs, 0);
    n.cubin(h, cubin->data());
    n.destroy(&h);
    std::lock_guard<std::mutex> lock(mu);
    cache[prog] = *cubin;
    return 0;
}

// Itanium name of the namespace-scope variable ns::name (what the module's
// symbol table holds for a __constant__ declared inside a namespace).
inline std::string hook_mangle(const char* ns, const std::string& name)
{
    return "_ZN" + std::to_string(strlen(ns)) + ns + std::to_string(name.size()) + name + "E";
}

inline std::string cu_error(CUresult r)
{
    const char* s = nullptr;
    if (drv().getErrorString) drv().getErrorString(r, &s);
    return s ? s : "CUDA driver error " + std::to_string((int)r);
}

// Load a compiled hook module into the current context and resolve its
// kernels and framework constants.
inline int hook_load(HookModule* h, const std::vector<char>& cubin, std::string* err)
{
    Driver& d = drv();
    if (!d.ok) {
        *err = "the CUDA driver API entry points are unavailable";
        return -2;
    }
    CUresult r = d.moduleLoadData(&h->mod, cubin.data());
    if (r != CUDA_SUCCESS) {
        *err = "cuModuleLoadData: " + cu_error(r);
        return -2;
    }
    const char* names[] = {"psh_prism32", "psh_prism64", "psh_gap32", "psh_gap64",
                           "psh_ybridge", "psh_octahedron", "psh_block"};
    CUfunction* dst[] = {&h->prism[0], &h->prism[1], &h->gap[0], &h->gap[1],
                         &h->ybridge,  &h->octahedron, &h->block};
    for (int i = 0; i < 7; ++i) {
        r = d.moduleGetFunction(dst[i], h->mod, names[i]);
        if (r == CUDA_SUCCESS)
            r = d.funcSetAttribute(*dst[i], CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES,
                                   227 * 1024);
        if (r != CUDA_SUCCESS) {
            *err = std::string(names[i]) + ": " + cu_error(r);
            return -2;
        }
    }
    for (int k = 0; k < 3; ++k)
        for (int f = 0; f < FW_COUNT; ++f) {
            size_t sz = 0;
            r = d.moduleGetGlobal(&h->fw[k][f], &sz, h->mod,
                                  hook_mangle(kHookNs[k], kHookFw[f]).c_str());
            if (r != CUDA_SUCCESS) {
                *err = std::string("framework constant ") + kHookFw[f] + ": " + cu_error(r);
                return -2;
            }
        }
    return 0;
}

// Find a user constant by name in the module (every namespace holds a copy);
// nullptr when the hook declares no such __constant__.
inline HookConst* hook_const(HookModule* h, const std::string& name)
{
    auto it = h->consts.find(name);
    if (it != h->consts.end()) return &it->second;
    for (int f = 0; f < FW_COUNT; ++f)
        if (name == kHookFw[f]) return nullptr;  // framework constants are not the plugin's
    HookConst c;
    for (int k = 0; k < 3; ++k) {
        size_t sz = 0;
        if (drv().moduleGetGlobal(&c.ptr[k], &sz, h->mod, hook_mangle(kHookNs[k], name).c_str()) !=
            CUDA_SUCCESS)
            return nullptr;
        c.size = sz;
    }
    auto ins = h->consts.emplace(name, c).first;
    ins->second.name = ins->first.c_str();
    return &ins->second;
}

// Write a framework constant of one namespace in stream order (skipped when
// it already holds the value).
inline CUresult hook_set_fw(HookModule* h, int ns, int f, int value, CUstream st)
{
    if (h->fw_val[ns][f] == value) return CUDA_SUCCESS;
    CUresult r = drv().memcpyHtoDAsync(h->fw[ns][f], &value, sizeof(int), st);
    if (r == CUDA_SUCCESS) h->fw_val[ns][f] = value;
    return r;
}

}  // namespace psb
