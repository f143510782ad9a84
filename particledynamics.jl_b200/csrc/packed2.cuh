// Two FP32 values in one 64-bit register pair: the packed multiply-add forms of sm_100 (one issue slot for two
// operations; each half rounds as the scalar instruction does).
#pragma once

#include <cuda_runtime.h>

namespace pdb {

struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 pk(float a) { return pk(a, a); }
// A constant pair that stays in its registers (every lane of the warp calls): a pair known to come from a kernel
// parameter, or to hold one value twice, is rebuilt by moves at every use; two shuffled values are not.
__device__ __forceinline__ f2 pk_held(float a) {
    return pk(__shfl_sync(0xffffffffu, a, 0), __shfl_sync(0xffffffffu, a, 1));
}
__device__ __forceinline__ void unpk(f2 x, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// 1 / sqrt(x) of a normal x (2 ulp, as rsqrtf; squared distances are never denormal).
__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 1 / x of a normal x: the hardware approximation (1 ulp) refined by one Newton-Raphson step, r + r (1 - x r).
__device__ __forceinline__ f2 rcp2(f2 x) {
    float a, b, ra, rb;
    unpk(x, a, b);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(a));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(b));
    const f2 r = pk(ra, rb), nr = pk(-ra, -rb);
    return fma2(r, fma2(x, nr, pk(1.f)), r);
}

}  // namespace pdb
