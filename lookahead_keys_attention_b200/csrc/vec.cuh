// Eight adjacent elements of a row as floats: one 16-byte access (two for fp32).
#pragma once
#include "sm100.cuh"

namespace castle {

template <typename T> struct Raw8 { uint4 q[sizeof(T) / 2]; };   // as they lie

template <typename T> __device__ __forceinline__ void load8(const T* p, float* v) {
  uint4 q = *reinterpret_cast<const uint4*>(p);
  const uint32_t* u = &q.x;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 f = Elem<T>::unpack2(u[j]);
    v[2 * j] = f.x; v[2 * j + 1] = f.y;
  }
}
template <> __device__ __forceinline__ void load8<float>(const float* p, float* v) {
  float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <typename T> __device__ __forceinline__ void store8(T* p, const float* v) {
  uint4 q;
  q.x = Elem<T>::pack2(v[0], v[1]); q.y = Elem<T>::pack2(v[2], v[3]);
  q.z = Elem<T>::pack2(v[4], v[5]); q.w = Elem<T>::pack2(v[6], v[7]);
  *reinterpret_cast<uint4*>(p) = q;
}
template <> __device__ __forceinline__ void store8<float>(float* p, const float* v) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

}  // namespace castle
