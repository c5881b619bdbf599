// Two FP32 values per register pair: the packed arithmetic of sm_100
// (add / sub / mul / fma .rn.f32x2), one instruction for both.  Each lane
// rounds as the scalar operation does.
#pragma once
#include <stdint.h>

namespace mxm {

struct f2 {
  unsigned long long v;
};
__device__ __forceinline__ f2 mk2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 dup2(float a) { return mk2(a, a); }
__device__ __forceinline__ void un2(f2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ f2 operator+(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator-(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 operator*(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// lane-wise scalar functions (no packed form exists)
template <class F>
__device__ __forceinline__ f2 each2(f2 x, F&& f) {
  float a, b;
  un2(x, a, b);
  return mk2(f(a), f(b));
}
template <class F>
__device__ __forceinline__ f2 each2(f2 x, f2 y, F&& f) {
  float a, b, c, d;
  un2(x, a, b);
  un2(y, c, d);
  return mk2(f(a, c), f(b, d));
}

}  // namespace mxm
