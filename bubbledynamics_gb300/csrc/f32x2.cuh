// Packed FP32 arithmetic (sm_100 and later).
#pragma once

namespace bd {

// Two cells as one 64-bit value: sm_103a's packed FP32 add, multiply
// and fma round each half like the scalar instruction and take one issue slot.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void f2_split(F2 a, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
// ptxas fuses a packed product into the packed add that takes it, although both
// are .rn: a product that goes into an add is formed by f2_mul1.
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// the product as two scalar multiplications
__device__ __forceinline__ F2 f2_mul1(F2 a, F2 b) {
    float a0, a1, b0, b1;
    f2_split(a, a0, a1);
    f2_split(b, b0, b1);
    return f2(__fmul_rn(a0, b0), __fmul_rn(a1, b1));
}
// a - b in one rounding (b (-1) + a)
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) { return f2_fma(b, f2(-1.0f), a); }
__device__ __forceinline__ F2 ld2(const float* p) {
    F2 r;
    r.v = *reinterpret_cast<const unsigned long long*>(p);
    return r;
}
__device__ __forceinline__ void st2(float* p, F2 a) { *reinterpret_cast<unsigned long long*>(p) = a.v; }

}  // namespace bd
