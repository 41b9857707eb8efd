// f32x2.cuh -- Blackwell's packed pairs of f32.
//
// A packed operation rounds each of its two lanes exactly like the scalar one.
// ptxas contracts a packed multiply whose only use is a packed add into a packed
// FMA, even with --fmad=false, which would round once instead of twice: a
// packed product (mul2) is only ever consumed by scalar adds (explicit .rn, never
// contracted), by further multiplies, or by conversions; a product for a packed
// add is fma2(a, b, negative_zeros()), which rounds as the product alone.
#pragma once
#include <cuda_runtime.h>

namespace mpm {
namespace x2 {

struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 x, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ float lo(f2 x) {
    float a, b;
    upk(x, a, b);
    return a;
}
__device__ __forceinline__ float hi(f2 x) {
    float a, b;
    upk(x, a, b);
    return b;
}
__device__ __forceinline__ f2 dup(float a) { return pk(a, a); }
__device__ __forceinline__ f2 neg2(f2 x) { return pk(-lo(x), -hi(x)); }
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
// Only for operands that are not packed products.
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}
// (-0, -0), from a number of the kernel's arguments that is never negative, so
// that ptxas cannot know it and take the addition out.
__device__ __forceinline__ f2 negative_zeros(int never_negative) {
    return dup(__int_as_float((int)(0x80000000u | (unsigned)never_negative >> 31)));
}

}  // namespace x2
}  // namespace mpm
