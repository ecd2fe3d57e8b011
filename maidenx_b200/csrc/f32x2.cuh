// Two f32 values in one 64-bit register pair: one instruction multiplies, adds or multiplies and adds both, each half rounded as the scalar instruction
// rounds it, so that arithmetic on 16-bit elements takes half the issue slots with the same results.
#pragma once

namespace mx {

struct F32x2 {
    unsigned long long v;
};
__device__ __forceinline__ F32x2 pair_of(float2 v) {
    F32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(v.x), "f"(v.y));
    return r;
}
__device__ __forceinline__ F32x2 twice(float v) { return pair_of(make_float2(v, v)); }
__device__ __forceinline__ float2 halves(F32x2 p) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p.v));
    return r;
}
__device__ __forceinline__ F32x2 operator*(F32x2 a, F32x2 b) {
    F32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F32x2 operator+(F32x2 a, F32x2 b) {
    F32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F32x2 fma2(F32x2 a, F32x2 b, F32x2 c) {
    F32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// gelu_f32_fast of both, bit for bit.
__device__ __forceinline__ float2 gelu_f32x2(float2 x) {
    const float k1 = -2.302208198f, k2 = -0.102943240f;
    const F32x2 xx = pair_of(x);
    const float2 arg = halves(xx * fma2(twice(k2), xx * xx, twice(k1)));
    float2 e;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(arg.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(arg.y));
    const float2 d = halves(twice(1.0f) + pair_of(e));
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
    return halves(xx * pair_of(r));
}

}  // namespace mx
