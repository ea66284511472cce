// Rotary embedding of a row, fused into the passes that read it (transform.cu, decode.cu).  Pairs of adjacent
// channels (2i, 2i+1) are rotated by position * freqs[i].  The rounding points are those of the element-wise torch
// form (castle.py, _Rotary.rotate): the angle in fp32, cosine, sine, both products and the sum rounded to the
// tensor's type, so both give the same bits.
#pragma once
#include "sm100.cuh"
#include "../../include/castle_b200.h"

namespace castle {

struct RotaryParams {
  const void* freqs;   // [dim_head / 2], null = no rotation
  int dtype;           // of freqs
  int inverse;         // rotate back (gradients)
  float position0;     // position of row 0
};

// Not inlined: the range reduction's slow path would cost the decode kernels registers in their main loop.
static __device__ __noinline__ float2 cos_sin(float angle) { return make_float2(cosf(angle), sinf(angle)); }

__device__ __forceinline__ float rotary_freq(const RotaryParams& r, int pair) {
  return r.dtype == CASTLE_F32 ? reinterpret_cast<const float*>(r.freqs)[pair]
         : r.dtype == CASTLE_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(r.freqs)[pair])
                                  : __half2float(reinterpret_cast<const __half*>(r.freqs)[pair]);
}
__device__ __forceinline__ float2 rotary_cos_sin(const RotaryParams& r, int n, float freq) {
  const float2 cs = cos_sin(__fmul_rn(__fadd_rn((float)n, r.position0), freq));
  return make_float2(cs.x, r.inverse ? -cs.y : cs.y);
}

template <typename T> __device__ __forceinline__ float round_to(float x) { return Elem<T>::to_f(Elem<T>::from_f(x)); }
template <> __device__ __forceinline__ float round_to<float>(float x) { return x; }

// One pair; cs = (cos, sin) unrounded.
template <typename T> __device__ __forceinline__ void rotate_pair(float& a, float& b, float2 cs) {
  const float c = round_to<T>(cs.x), s = round_to<T>(cs.y);
  const float x = round_to<T>(__fsub_rn(round_to<T>(__fmul_rn(a, c)), round_to<T>(__fmul_rn(b, s))));
  const float y = round_to<T>(__fadd_rn(round_to<T>(__fmul_rn(a, s)), round_to<T>(__fmul_rn(b, c))));
  a = x; b = y;
}
template <typename T> __device__ __forceinline__ void rotate8(float* v, const float2* cs) {
#pragma unroll
  for (int j = 0; j < 4; ++j) rotate_pair<T>(v[2 * j], v[2 * j + 1], cs[j]);
}

}  // namespace castle
