// Complex values (float2 / double2, or a pair of fixed-point integers) as the transforms use them.
#pragma once

namespace ocsc {

template <typename R> struct CT;
template <> struct CT<float> { using T = float2; };
template <> struct CT<double> { using T = double2; };
template <typename R> using Cx = typename CT<R>::T;

template <typename R> __host__ __device__ __forceinline__ Cx<R> cx(R a, R b) { Cx<R> c; c.x = a; c.y = b; return c; }
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> __device__ __forceinline__ C cmul(C a, C b) {
    C c; c.x = a.x * b.x - a.y * b.y; c.y = a.x * b.y + a.y * b.x; return c;
}
template <typename C> __device__ __forceinline__ C cconj(C a) { a.y = -a.y; return a; }
// multiply by -i (forward) or +i (inverse)
template <typename C> __device__ __forceinline__ C cmul_mi(C a) { C c; c.x = a.y; c.y = -a.x; return c; }
template <typename C> __device__ __forceinline__ C cmul_pi(C a) { C c; c.x = -a.y; c.y = a.x; return c; }

}  // namespace ocsc
