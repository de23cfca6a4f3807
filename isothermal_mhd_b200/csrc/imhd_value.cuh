// imhd_value.cuh -- the value types of the FP32 arithmetic: one single
// precision number (F1), or two of neighbouring cells or rows side by side in
// a 64-bit register pair (F2), with the same operators.
//
// The FP32 sweeps are bound by instruction issue, and one packed instruction
// (add/sub/mul/fma.rn.f32x2) does the work of two scalar ones in one issue
// slot; it takes the FP32 pipe as long as the two would.  Every operation on
// F1 and F2 is rounded separately and fused multiply-adds are written out
// (fma), so that the compiler contracts nothing by itself: the same expression
// gives the same bits in F1 and F2, in every kernel and in every copy that
// inlining makes.  That covers PLM.  The PPM edges and the primitive-variable
// limiters are written on plain floats (imhd_physics.cuh) in a unit compiled
// with contraction, and so are the FP64 eigenvector normalisations near the
// triple point: a column's first cells and its loop are separate copies of
// them, so FP32 PPM may differ in the last bit with the column length.
// What has no packed form (reciprocals, roots, minima, selections) runs on the
// halves.
#pragma once

#include <cuda_runtime.h>

namespace imhd {

struct F1 { float v; };
struct F2 { unsigned long long v; };

__device__ __forceinline__ F2 pack2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(F2 a, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}

template <class V> struct lanes_of { static constexpr int n = 1; };
template <> struct lanes_of<F2> { static constexpr int n = 2; };

__device__ __forceinline__ F1 operator+(F1 a, F1 b) { return F1{__fadd_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 operator-(F1 a, F1 b) { return F1{__fsub_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 operator*(F1 a, F1 b) { return F1{__fmul_rn(a.v, b.v)}; }
__device__ __forceinline__ F1 fma(F1 a, F1 b, F1 c) { return F1{__fmaf_rn(a.v, b.v, c.v)}; }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

template <class V> __device__ __forceinline__ V same(float a);
template <> __device__ __forceinline__ F1 same<F1>(float a) { return F1{a}; }
template <> __device__ __forceinline__ F2 same<F2>(float a) { return pack2(a, a); }

// f of each lane
template <class Fn> __device__ __forceinline__ F1 each(Fn f, F1 a) { return F1{f(a.v)}; }
template <class Fn> __device__ __forceinline__ F1 each(Fn f, F1 a, F1 b) { return F1{f(a.v, b.v)}; }
template <class Fn> __device__ __forceinline__ F1 each(Fn f, F1 a, F1 b, F1 c) { return F1{f(a.v, b.v, c.v)}; }
template <class Fn> __device__ __forceinline__ F2 each(Fn f, F2 a) {
    float x, y;
    unpack2(a, x, y);
    return pack2(f(x), f(y));
}
template <class Fn> __device__ __forceinline__ F2 each(Fn f, F2 a, F2 b) {
    float x, y, z, w;
    unpack2(a, x, y);
    unpack2(b, z, w);
    return pack2(f(x, z), f(y, w));
}
template <class Fn> __device__ __forceinline__ F2 each(Fn f, F2 a, F2 b, F2 c) {
    float x, y, z, w, s, t;
    unpack2(a, x, y);
    unpack2(b, z, w);
    unpack2(c, s, t);
    return pack2(f(x, z, s), f(y, w, t));
}
// lane l (0 or 1) and its replacement, for the rare per-lane branches
__device__ __forceinline__ float lane(F1 a, int) { return a.v; }
__device__ __forceinline__ float lane(F2 a, int l) {
    float x, y;
    unpack2(a, x, y);
    return l ? y : x;
}
__device__ __forceinline__ void set_lane(F1& a, int, float v) { a.v = v; }
__device__ __forceinline__ void set_lane(F2& a, int l, float v) {
    float x, y;
    unpack2(a, x, y);
    a = l ? pack2(x, v) : pack2(v, y);
}

template <class V> __device__ __forceinline__ V vrcp(V a) { return each([](float x) { return 1.0f / x; }, a); }
template <class V> __device__ __forceinline__ V vrsqrt(V a) { return each([](float x) { return rsqrtf(x); }, a); }
template <class V> __device__ __forceinline__ V vsqrt(V a) { return each([](float x) { return sqrtf(x); }, a); }
template <class V> __device__ __forceinline__ V vabs(V a) { return each([](float x) { return fabsf(x); }, a); }
template <class V> __device__ __forceinline__ V vmax2(V a, V b) { return each([](float x, float y) { return fmaxf(x, y); }, a, b); }
template <class V> __device__ __forceinline__ V vmin2(V a, V b) { return each([](float x, float y) { return fminf(x, y); }, a, b); }
// c >= 0 ? a : b
template <class V> __device__ __forceinline__ V vsel(V c, V a, V b) {
    return each([](float s, float x, float y) { return s >= 0.0f ? x : y; }, c, a, b);
}
// x with the sign of s
template <class V> __device__ __forceinline__ V vsign(float x, V s) {
    return each([x](float t) { return copysignf(x, t); }, s);
}
__device__ __forceinline__ bool any_less(F1 a, F1 b) { return a.v < b.v; }
__device__ __forceinline__ bool any_less(F2 a, F2 b) {
    float x, y, z, w;
    unpack2(a, x, y);
    unpack2(b, z, w);
    return x < z || y < w;
}
__device__ __forceinline__ float top_lane(F1 a) { return a.v; }
__device__ __forceinline__ float top_lane(F2 a) {
    float x, y;
    unpack2(a, x, y);
    return fmaxf(x, y);
}

// the larger lane; NaN when either is
__device__ __forceinline__ float nan_top(F2 a) {
    float x, y;
    unpack2(a, x, y);
    return x != x ? x : y != y ? y : fmaxf(x, y);
}

}  // namespace imhd
