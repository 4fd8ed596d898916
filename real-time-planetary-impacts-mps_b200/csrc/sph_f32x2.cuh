// sph_f32x2.cuh -- pairs of floats in the packed FP32 instructions of sm_100
// (add / mul / fma .rn.f32x2): one issue slot for two operations, each rounded
// as the scalar instruction rounds it.  The pair loops here are bound by issue
// slots and not by the FMA pipe, so they take two neighbours per step.
#pragma once

#include <cstdint>

namespace sph {

struct F2 {
    uint64_t v;
};

__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void unpack(F2 a, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ float sum(F2 a) {
    float x, y;
    unpack(a, x, y);
    return x + y;
}
__device__ __forceinline__ F2 neg(F2 a) { return F2{a.v ^ 0x8000000080000000ull}; }
__device__ __forceinline__ F2 clamp0(F2 a) {
    float x, y;
    unpack(a, x, y);
    return f2(fmaxf(x, 0.f), fmaxf(y, 0.f));
}
// The hardware's approximations (within 2 ulp), subnormal arguments taken as
// zero: one instruction each, where rsqrtf and __fdividef spend three to five
// more on arguments that are no distance or density here.
__device__ __forceinline__ float rsqrt_hw(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rcp_hw(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ F2 rsqrt2(F2 a) {
    float x, y;
    unpack(a, x, y);
    return f2(rsqrt_hw(x), rsqrt_hw(y));
}

}  // namespace sph
