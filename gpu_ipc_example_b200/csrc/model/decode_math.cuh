// Arithmetic that the decode-step kernels share: 16-bit pairs, the rotation of a pair, the warp-level tensor product of the
// attention, the order of the arg-max.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

namespace b200ipc {

constexpr int kAttnD = 128;  // head dimension of the attention kernels

template <typename T>
struct Num;
template <>
struct Num<__half> {
  using T2 = __half2;
  __device__ static float2 up(T2 v) { return __half22float2(v); }
  __device__ static T2 down(float a, float b) { return __floats2half2_rn(a, b); }
};
template <>
struct Num<__nv_bfloat16> {
  using T2 = __nv_bfloat162;
  __device__ static float2 up(T2 v) { return __bfloat1622float2(v); }
  __device__ static T2 down(float a, float b) { return __floats2bfloat162_rn(a, b); }
};

// Pair (x1, x2) turned by an angle.  Spelled out so that every kernel that rotates gives the same bits.
__device__ __forceinline__ float2 rope_pair(float x1, float x2, float sn, float cs) {
  return make_float2(fmaf(x1, cs, -__fmul_rn(x2, sn)), fmaf(x2, cs, __fmul_rn(x1, sn)));
}

template <typename T>
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1);
template <>
__device__ __forceinline__ void mma_16816<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                                  uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16816<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                         uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <typename T>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const typename Num<T>::T2 v = Num<T>::down(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Greatest value and where it stands: the first one of equal values; NaN is greater than everything.
struct Best {
  float v;
  int i;
};
__device__ __forceinline__ Best better(Best a, Best b) {
  const bool na = a.v != a.v, nb = b.v != b.v;
  const bool take_b = nb ? (!na || b.i < a.i) : (!na && (b.v > a.v || (b.v == a.v && b.i < a.i)));
  return take_b ? b : a;
}

}  // namespace b200ipc
