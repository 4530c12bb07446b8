// The heat equation's cell update and the storage types of its fields.
#pragma once
#include "swept.cuh"

namespace psb {

// Forward Euler in numpy's operation order (Heat in equations.cuh): centre c,
// rows xm above and xp below, columns ym left and yp right.
__device__ __forceinline__ double heat_fe(double c, double xm, double xp, double ym, double yp,
                                          double cr)
{
    const double dxx = __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, c, xp), xm));
    const double dyy = __dmul_rn(cr, __dadd_rn(__fma_rn(-2.0, c, yp), ym));
    return __dadd_rn(__dadd_rn(dxx, dyy), c);
}

// Storage type of the fields.  double; or float, every level evaluated in
// double and rounded to float (the reference's float32 runs: its courant is a
// float64 scalar, so numpy computes each level in float64 and rounds it when
// it is stored).  Registers and arithmetic are double in both cases.
template <class T>
struct Pair2;
template <>
struct Pair2<double> {
    using type = double2;
};
template <>
struct Pair2<float> {
    using type = float2;
};

template <class T>
__device__ __forceinline__ double to_level(double x)
{
    return x;
}
template <>
__device__ __forceinline__ double to_level<float>(double x)
{
    return (double)__double2float_rn(x);
}

template <class T>
__device__ __forceinline__ typename Pair2<T>::type pair2(double x, double y);
template <>
__device__ __forceinline__ double2 pair2<double>(double x, double y)
{
    return make_double2(x, y);
}
template <>
__device__ __forceinline__ float2 pair2<float>(double x, double y)
{
    return make_float2((float)x, (float)y);  // exact: x, y already carry float precision
}

template <class P>
__device__ __forceinline__ double2 widen(P v)
{
    return make_double2((double)v.x, (double)v.y);
}

// one pair of T (16 bytes for double, 8 for float)
template <class T>
__device__ __forceinline__ void cp_async_pair(T* smem, const T* gmem)
{
    if constexpr (sizeof(T) == 8)
        cp_async16(smem, gmem);
    else
        cp_async8(smem, gmem);
}

}  // namespace psb
