// Two floats in an aligned register pair: one instruction of the FMA pipe does both halves, each rounded by itself as the
// instruction on one float rounds it.  It saves issue slots, not time of the pipe, which takes a pair as two: it pays where other
// instructions of the same warps wait for slots (the softmax of attention_tcgen05.cu), not where FMAs are all there is (the scan
// of state_scan.cu in pairs: 291 -> 295 us).
#pragma once

typedef unsigned long long f32x2;          // the low half: the first float

__device__ __forceinline__ f32x2 pack2(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ f32x2 twice(float x) { return pack2(x, x); }
__device__ __forceinline__ void unpack2(f32x2 v, float& x, float& y) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(x), "=f"(y) : "l"(v)); }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
