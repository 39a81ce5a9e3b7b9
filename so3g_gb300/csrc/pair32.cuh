// pair32.cuh -- two float32 values in a register pair, operated on by one
// instruction (f32x2, sm_100 and later).  Each half is rounded as the scalar
// operation's result; the kernels whose bound is the rate of instruction
// issue use them where two values go through the same steps.
#pragma once

namespace so3g {

struct f32x2 {
    unsigned long long b;
};

__device__ __forceinline__ f32x2 f2_make(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.b) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ f32x2 f2_both(float x) { return f2_make(x, x); }
__device__ __forceinline__ void f2_get(f32x2 a, float &x, float &y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.b));
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ f32x2 f2_sub(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(a.b), "l"(b.b));
    return r;
}
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(a.b), "l"(b.b), "l"(c.b));
    return r;
}

// Knuth's TwoSum of each half: s + e == a + b exactly.
__device__ __forceinline__ void f2_two_sum(f32x2 a, f32x2 b, f32x2 &s, f32x2 &e) {
    s = f2_add(a, b);
    const f32x2 bb = f2_sub(s, a);
    e = f2_add(f2_sub(a, f2_sub(s, bb)), f2_sub(b, bb));
}

}  // namespace so3g
