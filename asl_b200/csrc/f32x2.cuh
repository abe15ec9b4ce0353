// Two FP32 values in one 64-bit register pair, for the packed FP32
// instructions of sm_100 (fma / add / sub .f32x2): each half is rounded
// exactly as the scalar instruction rounds it, so a collision evaluated on a
// pair of cells gives both cells the bits that the scalar one gives, in half
// the instructions. Division and square root stay scalar, per half.
#pragma once
#include <cuda_runtime.h>

namespace aslb {

struct F2 {
  unsigned long long v;
  F2() = default;
  __device__ __forceinline__ F2(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi)); }
  __device__ __forceinline__ F2(float both) : F2(both, both) {}
  __device__ __forceinline__ explicit F2(double both) : F2(float(both)) {}
  __device__ __forceinline__ explicit F2(int both) : F2(float(both)) {}
  __device__ __forceinline__ float lo() const {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    (void)b;
    return a;
  }
  __device__ __forceinline__ float hi() const {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    (void)a;
    return b;
  }
};

// A product is a multiply-add with -0 (the same bits for every product, its
// zeros included): a packed multiply feeding a packed add may be contracted
// into one multiply-add, explicit rounding or not, which rounds once less.
__device__ __forceinline__ F2 mul_(F2 a, F2 b) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(0x8000000080000000ull));
  return r;
}
__device__ __forceinline__ F2 add_(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 sub_(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma_(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 div_(F2 a, F2 b) { return F2(__fdiv_rn(a.lo(), b.lo()), __fdiv_rn(a.hi(), b.hi())); }
__device__ __forceinline__ F2 sqrt_(F2 a) { return F2(__fsqrt_rn(a.lo()), __fsqrt_rn(a.hi())); }
__device__ __forceinline__ F2 operator-(F2 a) { return F2(-a.lo(), -a.hi()); }

}  // namespace aslb
