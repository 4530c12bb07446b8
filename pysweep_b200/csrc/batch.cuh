// Batched swept phases: many independent instances (uneven grid sizes) advance
// together, one launch per phase for all of them.
//
// Every instance has two descriptors (SweptArgs for even and odd
// half-cycles: base buffers swapped, prism bands offset by 0 or bs/2) and
// contributes its (band, segment) units to one flat unit table of
// (instance, unit) pairs.  A batched launch maps warp / CTA g to table entry g
// and runs the same body as the single-instance kernel.  All instances share
// the blocksize, so they share the levels per half-cycle and the shared-memory
// layout.  The launches of a whole run are captured into one CUDA graph.
// (Heat with forward Euler runs in the overlapped blocks' batched kernels,
// heat_block.cuh, Euler in the marching warps', euler_march.cuh.)
#pragma once
#include "swept.cuh"

namespace psb {

// Descriptors [instance][role][parity]: role 0 for the prism stream and the
// y-bridge, role 1 for the gap stream and the octahedron (their y-faces live in
// a second buffer, because the gap runs beside the y-bridge).  The kernels
// keep a copy in registers, with this launch's levels and first level.
template <bool GAP>
__device__ __forceinline__ void batch_args(const SweptArgs* __restrict__ desc, int inst,
                                           int parity, int H, long long L0, SweptArgs& a)
{
    a = desc[4 * inst + 2 * (GAP ? 1 : 0) + parity];
    a.H = H;
    a.L0 = L0;
}

// The generic batched kernels hold the descriptor fields in registers (the
// single-instance kernels read them from the parameter bank), so they are
// capped at the single-instance register budget to keep two stream CTAs (four
// seam CTAs) per SM.
template <class Eq, int ITS, int W, bool GAP, int NT>
__global__ void __launch_bounds__(NT, 2)
    stream_batch(const SweptArgs* __restrict__ desc, const int2* __restrict__ units, int parity,
                 int H, long long L0)
{
    extern __shared__ double sm[];
    const int2 u = units[blockIdx.x];
    SweptArgs a;
    batch_args<GAP>(desc, u.x, parity, H, L0, a);
    stream_body<Eq, ITS, W, GAP, NT>(a, u.y, sm);
}

template <class Eq, int ITS, bool GAP, int NT>
__global__ void __launch_bounds__(NT, 4)
    seam_batch(const SweptArgs* __restrict__ desc, const int2* __restrict__ units, int parity,
               int H, long long L0)
{
    extern __shared__ double sm[];
    const int2 u = units[blockIdx.x];
    SweptArgs a;
    batch_args<GAP>(desc, u.x, parity, H, L0, a);
    seam_body<Eq, ITS, GAP, NT>(a, u.y, sm);
}

}  // namespace psb
