// sph_pack.cuh -- packed FP32 arithmetic: two values per instruction (add, mul
// and fma .f32x2), each rounded as the scalar operation would be.
#pragma once

#include "sph_device.cuh"

namespace sph {

struct F2 {
    unsigned long long v;
    __device__ __forceinline__ float lo() const {
        float a;
        asm("mov.b64 {%0, _}, %1;" : "=f"(a) : "l"(v));
        return a;
    }
    __device__ __forceinline__ float hi() const {
        float b;
        asm("mov.b64 {_, %0}, %1;" : "=f"(b) : "l"(v));
        return b;
    }
};
__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
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

}  // namespace sph
