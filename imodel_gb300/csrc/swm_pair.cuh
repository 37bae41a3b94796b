// Arithmetic of the FP32 stage over one value or over two members' values at
// once (internal header).
//
// Two members of an ensemble share a tile's records, indices and addresses,
// and sm_103a does two FP32 operations in one instruction on a pair of
// registers (fma/mul/add .f32x2, each half rounded as the single operation):
// the pair takes about as many instructions as one member.
#pragma once
#include <cstdint>

namespace imodel {

struct alignas(8) Pair {
  float x, y;
};

namespace pair_detail {
__device__ __forceinline__ unsigned long long bits(Pair a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ Pair pair(unsigned long long r) {
  Pair a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
}  // namespace pair_detail

// V where it is not deduced (a null pointer may stand for V *)
template <class V>
struct ValueOf {
  using type = V;
};

// one value for all members
template <class V>
__device__ __forceinline__ V all(float a);
template <>
__device__ __forceinline__ float all<float>(float a) {
  return a;
}
template <>
__device__ __forceinline__ Pair all<Pair>(float a) {
  return Pair{a, a};
}

__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
// the same where no fused operation can arise: the compiler schedules plain
// operators better than the intrinsics (level 7 38.9 -> 37.2 us a step)
__device__ __forceinline__ float padd(float a, float b) { return a + b; }
__device__ __forceinline__ float pmul(float a, float b) { return a * b; }
__device__ __forceinline__ float psub(float a, float b) { return a - b; }
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ Pair vfma(Pair a, Pair b, Pair c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(pair_detail::bits(a)), "l"(pair_detail::bits(b)), "l"(pair_detail::bits(c)));
  return pair_detail::pair(r);
}
__device__ __forceinline__ Pair vmul(Pair a, Pair b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(pair_detail::bits(a)), "l"(pair_detail::bits(b)));
  return pair_detail::pair(r);
}
__device__ __forceinline__ Pair vadd(Pair a, Pair b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(r)
      : "l"(pair_detail::bits(a)), "l"(pair_detail::bits(b)));
  return pair_detail::pair(r);
}
__device__ __forceinline__ Pair vneg(Pair a) { return Pair{-a.x, -a.y}; }
// a - b = a + (-1) b: the product is exact
__device__ __forceinline__ Pair vsub(Pair a, Pair b) { return vfma(all<Pair>(-1.0f), b, a); }
__device__ __forceinline__ Pair padd(Pair a, Pair b) { return vadd(a, b); }
__device__ __forceinline__ Pair pmul(Pair a, Pair b) { return vmul(a, b); }
__device__ __forceinline__ Pair psub(Pair a, Pair b) { return vsub(a, b); }

}  // namespace imodel
