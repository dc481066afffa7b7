#pragma once

namespace ske {

// Packed pairs of floats for the f32x2 instructions: two independent IEEE
// operations, round to nearest, no flush to zero.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1,%2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) { asm("mov.b64 {%0,%1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// (s, t) with s = fl(a + b) and t the exact rest (Knuth's two-sum).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& t) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    t = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// A float32 sum with its roundings carried along.
struct CarriedSum {
    float sum = 0.0f, rest = 0.0f;
    __device__ __forceinline__ void add(float v) {
        float s, t;
        two_sum(sum, v, s, t);
        sum = s;
        rest += t;
    }
    __device__ __forceinline__ void add(float2 v) {
        add(v.x);
        rest += v.y;
    }
    // (The rest of an infinite sum is NaN.)
    __device__ __forceinline__ float value() const { return isfinite(sum) ? sum + rest : sum; }
};

}  // namespace ske
