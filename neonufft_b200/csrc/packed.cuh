// Packed arithmetic on pairs of values (fma.rn.f32x2 in single precision) and the atomic adds of
// cells, shared by the register-window kernels (zwin.cu, strip.cu).
#pragma once

#include "common.cuh"

namespace nnb {

template <typename T>
struct Packed;

template <>
struct Packed<float> {
  using P = unsigned long long;  // two floats in one 64-bit register pair
  static __device__ __forceinline__ P zero() { return 0ull; }
  static __device__ __forceinline__ P pack(float x, float y) {
    P r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
  }
  static __device__ __forceinline__ P splat(float x) { return pack(x, x); }
  static __device__ __forceinline__ float lo(P v) {
    float x;
    asm("mov.b64 {%0, _}, %1;" : "=f"(x) : "l"(v));
    return x;
  }
  static __device__ __forceinline__ float hi(P v) {
    float y;
    asm("mov.b64 {_, %0}, %1;" : "=f"(y) : "l"(v));
    return y;
  }
  static __device__ __forceinline__ P shfl(P v, int lane) {
    return __shfl_sync(0xffffffffu, v, lane);
  }
  // a * b + c, elementwise
  static __device__ __forceinline__ P fma(P a, P b, P c) {
    P d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
  }
  static __device__ __forceinline__ P add(P a, P b) {
    P d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
  }
};

template <>
struct Packed<double> {
  using P = double2;
  static __device__ __forceinline__ P zero() { return P{0.0, 0.0}; }
  static __device__ __forceinline__ P pack(double x, double y) { return P{x, y}; }
  static __device__ __forceinline__ P splat(double x) { return P{x, x}; }
  static __device__ __forceinline__ double lo(P v) { return v.x; }
  static __device__ __forceinline__ double hi(P v) { return v.y; }
  static __device__ __forceinline__ P shfl(P v, int lane) {
    return P{__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane)};
  }
  static __device__ __forceinline__ P fma(P a, P b, P c) {
    return P{::fma(a.x, b.x, c.x), ::fma(a.y, b.y, c.y)};
  }
  static __device__ __forceinline__ P add(P a, P b) { return P{a.x + b.x, a.y + b.y}; }
};

// Four consecutive values of a 16-byte aligned shared-memory array as two pairs.
template <typename T>
__device__ __forceinline__ void load_pairs(const T* p, typename Packed<T>::P* k);
template <>
__device__ __forceinline__ void load_pairs<float>(const float* p, unsigned long long* k) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  k[0] = v.x;
  k[1] = v.y;
}
template <>
__device__ __forceinline__ void load_pairs<double>(const double* p, double2* k) {
  k[0] = *reinterpret_cast<const double2*>(p);
  k[1] = *reinterpret_cast<const double2*>(p + 2);
}

__device__ __forceinline__ void atomic_add_cplx(float2* p, float2 v) { atomicAdd(p, v); }
__device__ __forceinline__ void atomic_add_cplx(double2* p, double2 v) {
  atomicAdd(&p->x, v.x);
  atomicAdd(&p->y, v.y);
}

// Adds two neighbouring cells (re0, im0), (re1, im1) at a 16-byte aligned address.
__device__ __forceinline__ void atomic_add_pair(float2* p, float re0, float im0, float re1,
                                                float im1) {
  atomicAdd(reinterpret_cast<float4*>(p), make_float4(re0, im0, re1, im1));
}
__device__ __forceinline__ void atomic_add_pair(double2* p, double re0, double im0, double re1,
                                                double im1) {
  atomic_add_cplx(p, double2{re0, im0});
  atomic_add_cplx(p + 1, double2{re1, im1});
}

}  // namespace nnb
