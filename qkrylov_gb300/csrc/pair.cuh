// FP32 arithmetic on (re, im) pairs held in 64 bits: one instruction for both halves
// (fma / mul / add .f32x2), each rounded as its scalar counterpart.
#pragma once

namespace qkg {
namespace pairk {
using u64 = unsigned long long;

__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 pk(float x, float y) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
    return d;
}
__device__ __forceinline__ float2 unpk(u64 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
constexpr u64 kMinusOne2 = 0xBF800000BF800000ull;  // (-1, -1)
__device__ __forceinline__ u64 sub2(u64 a, u64 b) { return fma2(b, kMinusOne2, a); }  // a - b, rounded once
// (hi, lo) += a * b elementwise, compensated (TwoProduct, TwoSum), both halves at once
__device__ __forceinline__ void acc2(u64& hi, u64& lo, u64 a, u64 b) {
    const u64 p = mul2(a, b);
    const u64 e = fma2(a, b, mul2(p, kMinusOne2));
    const u64 t = add2(hi, p);
    const u64 z = sub2(t, hi);
    const u64 err = add2(sub2(hi, sub2(t, z)), sub2(p, z));
    lo = add2(lo, add2(err, e));
    hi = t;
}

}  // namespace pairk
}  // namespace qkg
