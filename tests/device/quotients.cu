// The marching warps' reciprocals and quotients (euler_march.cuh) against CUDA's
// correctly rounded operations, bit for bit, over their safe ranges.  Built and
// run by tests/test_gpu_euler_quotients.py.  Prints the number of pairs compared
// and of results that differ, of each function.
#include <cstdio>

#include "../../pysweep_b200/csrc/euler_march.cuh"

using namespace psb;

struct Count {
    unsigned long long pairs, recip, quot, quots;
};

__device__ unsigned long long mix(unsigned long long x)  // splitmix64
{
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// 2^e with the 52 mantissa bits m
__device__ double number(unsigned long long m, int e)
{
    return __longlong_as_double((long long)((unsigned long long)(e + 1023) << 52 | (m & 0xfffffffffffffull)));
}

// mantissas: uniform, or a few ulps above or below a power of two or three halves
__device__ unsigned long long mantissa(unsigned long long h)
{
    const unsigned long long k = (h >> 8) & 15;
    switch (h & 7) {
    case 0: return k;
    case 1: return 0xfffffffffffffull - k;
    case 2: return 0x8000000000000ull + k - 8;
    case 3: return 1ull << (h >> 20 & 63) % 52;
    default: return mix(h);
    }
}

__device__ void compare(double a, double b, Count& c)
{
    const euler::Recip r = euler::recip(b);
    const double q = __ddiv_rn(a, b), one[2] = {a, -a};
    double two[2];
    euler::quots(one, r, two);
    // (a quotient that is zero has either sign: quot returns +0)
    auto differ = [](double x, double y) {
        return x != y || (x != 0.0 && __double_as_longlong(x) != __double_as_longlong(y));
    };
    ++c.pairs;
    c.recip += differ(r.y, __drcp_rn(b)) || differ(euler::recip_rn(b), __drcp_rn(b));
    c.quot += differ(euler::quot(a, r), q);
    c.quots += differ(two[0], q) || differ(two[1], -q);
}

// b: 2^-80 .. 2^80, its ends included; a: zero, 2^-930 .. 2^245, or one whose
// quotient lies next to a midpoint of two doubles
__global__ void check(unsigned long long seed, int n, Count* out)
{
    Count c = {0, 0, 0, 0};
    const unsigned long long id = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (int i = 0; i < n; ++i) {
        const unsigned long long h = mix(seed ^ mix(id * n + i)), g = mix(h), k = mix(g);
        const int eb = (h >> 32) % 32 == 0 ? ((h >> 40 & 1) ? 79 : -80) : (int)((h >> 32) % 160) - 80;
        const double b = number(mantissa(h), eb);
        const double sign = (g & 1) ? -1.0 : 1.0;
        double a = number(mantissa(g >> 1), (int)((g >> 32) % 1175) - 930);
        if (k % 16 == 0) a = 0.0;
        compare(sign * a, b, c);
        compare(sign * b, b, c);
        compare(sign, b, c);
        // quotients that all but tie: for the odd integer B of 53 bits and an odd
        // M = r / B mod 2^54 of 54 bits, A = (B M - r) / 2^54 is an integer and
        // A / B = (M - r/B) / 2^54, next to the midpoint M
        const unsigned long long B = 1ull << 52 | (k & 0xfffffffffffffull) | 1;
        unsigned long long inv = B;
        for (int s = 0; s < 6; ++s) inv *= 2 - B * inv;
        for (int r = -3; r <= 3; r += 2) {
            const unsigned long long M = inv * (unsigned long long)(long long)r & ((1ull << 54) - 1);
            if (M < 1ull << 53) continue;
            unsigned long long lo = B * M, top = __umul64hi(B, M);
            const unsigned long long sub = (unsigned long long)(long long)r;
            top -= (r < 0 ? ~0ull : 0) + (lo < sub);
            lo -= sub;
            compare(sign * (double)(top << 10 | lo >> 54), (double)B, c);
            compare(sign * (double)(top << 10 | lo >> 54) * 0x1p-100, (double)B * 0x1p-130, c);
        }
    }
    atomicAdd(&out->pairs, c.pairs);
    atomicAdd(&out->recip, c.recip);
    atomicAdd(&out->quot, c.quot);
    atomicAdd(&out->quots, c.quots);
}

int main()
{
    Count *d, h;
    if (cudaMalloc(&d, sizeof h) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof h);
    check<<<592, 256>>>(20240817, 1024, d);
    if (cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
    printf("%llu %llu %llu %llu\n", h.pairs, h.recip, h.quot, h.quots);
    return 0;
}
