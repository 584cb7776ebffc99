// Packed FP32 pairs (Blackwell f32x2 instructions, sm_100 and later): two lanes of a 64-bit
// register hold the same quantity for two items, so one instruction serves both.
#pragma once

namespace fg {

using u64 = unsigned long long;
__device__ __forceinline__ u64 pk2(float lo, float hi) {
    u64 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ void upk2(u64 v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
    u64 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
    u64 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
    u64 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
    u64 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ u64 neg2(u64 a) { return a ^ 0x8000000080000000ull; }

// Double-single pairs, the operations of fg_ds.cuh lane by lane.
struct ds2 { u64 h, l; };
__device__ __forceinline__ ds2 ds2_quick(u64 a, u64 b) {
    const u64 s = add2(a, b);
    return {s, sub2(b, sub2(s, a))};
}
__device__ __forceinline__ ds2 ds2_two_sum(u64 a, u64 b) {
    const u64 s = add2(a, b), bb = sub2(s, a);
    return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ ds2 ds2_add(ds2 x, ds2 y) {
    const ds2 s = ds2_two_sum(x.h, y.h);
    return ds2_quick(s.h, add2(s.l, add2(x.l, y.l)));
}
__device__ __forceinline__ ds2 ds2_mul(ds2 x, ds2 y) {
    const u64 p = mul2(x.h, y.h);
    u64 e = fma2(x.h, y.h, neg2(p));
    e = fma2(x.h, y.l, e);
    e = fma2(x.l, y.h, e);
    return ds2_quick(p, e);
}

}  // namespace fg
