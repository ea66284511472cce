// What the cached-step kernels (decode.cu, token_layer.cu, token_linear.cu) share: 16-byte vectors of a row as floats, the sums over the
// lanes of a row, the rotation of the new rows.
#pragma once
#include "rotary.cuh"
#include "sm100.cuh"

namespace castle {

template <typename T> struct Vec;  // 16 bytes of T <-> floats
template <> struct Vec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(uint4 q, float* v) {
    v[0] = __uint_as_float(q.x); v[1] = __uint_as_float(q.y); v[2] = __uint_as_float(q.z); v[3] = __uint_as_float(q.w);
  }
  static __device__ __forceinline__ void load(const float* p, float* v) { unpack(*reinterpret_cast<const uint4*>(p), v); }
  static __device__ __forceinline__ void store(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
  static __device__ __forceinline__ void round(float*) {}
};
template <typename T> struct Vec16 {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(uint4 q, float* v) {
    float2 a = Elem<T>::unpack2(q.x), b = Elem<T>::unpack2(q.y), c = Elem<T>::unpack2(q.z), d = Elem<T>::unpack2(q.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
  static __device__ __forceinline__ void load(const T* p, float* v) { unpack(*reinterpret_cast<const uint4*>(p), v); }
  static __device__ __forceinline__ void store(T* p, const float* v) {
    uint4 q;
    q.x = Elem<T>::pack2(v[0], v[1]); q.y = Elem<T>::pack2(v[2], v[3]);
    q.z = Elem<T>::pack2(v[4], v[5]); q.w = Elem<T>::pack2(v[6], v[7]);
    *reinterpret_cast<uint4*>(p) = q;
  }
  // round to the storage type, so the value used for the score equals the value stored
  static __device__ __forceinline__ void round(float* v) {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = Elem<T>::to_f(Elem<T>::from_f(v[i]));
  }
};
template <> struct Vec<__nv_bfloat16> : Vec16<__nv_bfloat16> {};
template <> struct Vec<__half> : Vec16<__half> {};

__device__ __forceinline__ float sigmoid_f(float x) { return 1.f / (1.f + __expf(-x)); }

template <int LPR>
__device__ __forceinline__ float group_sum(float v) {
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The new token's rows are rotated as they are loaded: VEC adjacent elements of a row from column `col`.
template <typename T>
__device__ __forceinline__ void rotate_new(const RotaryParams& r, int64_t col, float* a, float* b, float* c) {
  if (r.freqs == nullptr) return;
  float f[Vec<T>::N / 2];
#pragma unroll
  for (int i = 0; i < Vec<T>::N / 2; ++i) f[i] = rotary_freq(r, (int)col / 2 + i);
#pragma unroll
  for (int i = 0; i < Vec<T>::N; i += 2) {
    const float2 cs = rotary_cos_sin(r, 0, f[i / 2]);
    rotate_pair<T>(a[i], a[i + 1], cs);
    rotate_pair<T>(b[i], b[i + 1], cs);
    if (c) rotate_pair<T>(c[i], c[i + 1], cs);
  }
}

}  // namespace castle
