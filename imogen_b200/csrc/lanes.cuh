// Lanes of the segment and window kernels: the same arithmetic on one number (FP32 or FP64), or on two
// independent FP32 numbers packed in a register pair.  Blackwell adds, multiplies and FMAs such a pair
// with one instruction; measured on a B200, the packed forms issue at half the rate of the scalar ones
// (1.9 against 3.6 warp instructions per clock and SM), i.e. the same operations per clock from half
// the issue slots, which the FP64, conversion, comparison and memory instructions beside them can use.
#pragma once

#include "common.cuh"

namespace img {

struct F2 {
    unsigned long long v;
    __device__ __forceinline__ F2() {}
    __device__ __forceinline__ F2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ void get(float& a, float& b) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
};
__device__ __forceinline__ F2 v_add(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 v_mul(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 v_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 v_sub(F2 a, F2 b) { return v_fma(b, F2(-1.f, -1.f), a); }   // exact product
template <typename T> __device__ __forceinline__ T v_add(T a, T b) { return a + b; }
template <typename T> __device__ __forceinline__ T v_mul(T a, T b) { return a * b; }
template <typename T> __device__ __forceinline__ T v_sub(T a, T b) { return a - b; }
__device__ __forceinline__ float v_fma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double v_fma(double a, double b, double c) { return fma(a, b, c); }
template <typename V> __device__ __forceinline__ V v_splat(double x) { return (V)x; }
template <> __device__ __forceinline__ F2 v_splat<F2>(double x) { return F2((float)x, (float)x); }

template <typename V, typename T> __device__ __forceinline__ V v_dup(T x) {
    if constexpr (sizeof(V) != sizeof(T)) return V(x, x);
    else return x;
}

__device__ __forceinline__ F2 v_pick(bool c, F2 a, F2 b) { a.v = c ? a.v : b.v; return a; }
template <typename T> __device__ __forceinline__ T v_pick(bool c, T a, T b) { return c ? a : b; }

// The limiter correction of each lane.  Van Leer: dL dR / (dL + dR) where the product is positive, else 0.
// A positive FP32 product keeps |dL + dR| above 2^-75, so the one-instruction reciprocal never sees a
// subnormal (which its .ftz form would flush).  The maximum with 0 takes negative products and NaN (both
// overflow: inf * 0), as limiter_corr_t does; the sign of the sum follows.
__device__ __forceinline__ float vanleer_part(float p, float s) { return copysignf(fmaxf(p * rcp_ftz(fabsf(s)), 0.f), s); }
template <int LIM>
__device__ __forceinline__ float v_limit(float dL, float dR) {
    if constexpr (LIM == LIM_VANLEER) return vanleer_part(dL * dR, dL + dR);
    else return limiter_corr_t<LIM>(dL, dR);
}
template <int LIM>
__device__ __forceinline__ F2 v_limit(F2 dL, F2 dR) {
    if constexpr (LIM == LIM_VANLEER) {
        float p0, p1, s0, s1;
        v_mul(dL, dR).get(p0, p1);
        v_add(dL, dR).get(s0, s1);
        return F2(vanleer_part(p0, s0), vanleer_part(p1, s1));
    } else {
        float l0, l1, r0, r1;
        dL.get(l0, l1);
        dR.get(r0, r1);
        return F2(limiter_corr_t<LIM>(l0, r0), limiter_corr_t<LIM>(l1, r1));
    }
}
template <int LIM>
__device__ __forceinline__ double v_limit(double dL, double dR) { return limiter_corr_t<LIM>(dL, dR); }

}  // namespace img
