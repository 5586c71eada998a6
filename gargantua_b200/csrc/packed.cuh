// Two FP32 values in a register pair, and the packed f32x2 instructions of
// sm_100 on them: each half is rounded as the scalar instruction rounds. One
// takes one issue slot and two cycles of the FMA pipe (measured: 2.06 cycles
// a warp; a scalar fma 1.1, 1.4 with a literal constant), so packing pays
// where the issue slots bound a kernel. Min, max, selects, reciprocals and
// square roots have no packed form.
#pragma once

#include "common.cuh"

namespace gg {

struct F2 {
    unsigned long long v;
};

__device__ __forceinline__ F2 f2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 parts(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}

__device__ __forceinline__ F2 mad(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 minus(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

}  // namespace gg
