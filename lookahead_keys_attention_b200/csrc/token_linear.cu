// y = norm(x) @ w^T for the handful of rows a cached single-token step projects (one row per sequence).
//
// At this size the product is a stream over the weights, and what a library call costs is its host side: one RMSNorm
// and two linear calls took 30 us of the 36 us a bf16 token's layer took on the host, for 9 us of kernels.  Here the
// norm is folded into the projection (every CTA computes it from x, which it needs whole anyway) and a call is one
// launch.  A warp owns WR rows of w and streams them with 16-byte loads; x sits in shared memory as fp32; all sums are
// fp32.  At 1 x 512 -> 3072 -> 512 bf16 the kernels take 2.8 and 2.3 us where the library calls took 2.7 + 3.8 and 3.0.
#include "common.cuh"
#include "sm100.cuh"

namespace castle {

constexpr int kTokenThreads = 128;
constexpr int kTokenSmem = 96 * 1024;   // x as fp32

template <typename T> struct Wide;      // 16 bytes of T
template <> struct Wide<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void unpack(uint4 q, float* v) {
    v[0] = __uint_as_float(q.x); v[1] = __uint_as_float(q.y); v[2] = __uint_as_float(q.z); v[3] = __uint_as_float(q.w);
  }
  static __device__ __forceinline__ float round(float x) { return x; }
  static __device__ __forceinline__ float cast(float x) { return x; }
};
template <typename T> struct Wide {
  static constexpr int N = 8;
  static __device__ __forceinline__ void unpack(uint4 q, float* v) {
    const float2 a = Elem<T>::unpack2(q.x), b = Elem<T>::unpack2(q.y), c = Elem<T>::unpack2(q.z), d = Elem<T>::unpack2(q.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
  static __device__ __forceinline__ float round(float x) { return Elem<T>::to_f(Elem<T>::from_f(x)); }
  static __device__ __forceinline__ T cast(float x) { return Elem<T>::from_f(x); }
};

struct TokenLinearParams {
  const void *x, *norm, *w;
  void* y;
  int rows, K, N;
  int64_t ldx;
  float eps;
};

// R = rows of x (padded up to 1, 2, 4 or 8), WR = rows of w per warp.
template <typename T, int R, int WR>
__global__ void __launch_bounds__(kTokenThreads) castle_token_linear_kernel(const TokenLinearParams p) {
  constexpr int V = Wide<T>::N, NW = kTokenThreads / 32;
  extern __shared__ __align__(16) float xs[];   // [R][K]
  __shared__ float part[NW][R];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = (blockIdx.x * NW + warp) * WR;
  const int chunks = p.K / V;
  const uint4* wrow[WR];
#pragma unroll
  for (int i = 0; i < WR; ++i)
    wrow[i] = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.w) + (int64_t)min(n0 + i, p.N - 1) * p.K);
  uint4 q[WR];   // the first chunk of the weights is on its way while x is prepared
  if (lane < chunks) {
#pragma unroll
    for (int i = 0; i < WR; ++i) q[i] = wrow[i][lane];
  }
  float ss[R];
#pragma unroll
  for (int r = 0; r < R; ++r) ss[r] = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + (int64_t)min(r, p.rows - 1) * p.ldx);
    for (int c = threadIdx.x; c < chunks; c += kTokenThreads) {
      float v[V];
      Wide<T>::unpack(src[c], v);
#pragma unroll
      for (int j = 0; j < V; ++j) { ss[r] = fmaf(v[j], v[j], ss[r]); xs[r * p.K + c * V + j] = v[j]; }
    }
  }
  if (p.norm) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
      if (lane == 0) part[warp][r] = ss[r];
    }
    __syncthreads();
    const uint4* nw = reinterpret_cast<const uint4*>(p.norm);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      float s = part[0][r];
#pragma unroll
      for (int k = 1; k < NW; ++k) s += part[k][r];
      const float inv = rsqrtf(s / (float)p.K + p.eps);
      for (int c = threadIdx.x; c < chunks; c += kTokenThreads) {   // the thread's own elements
        float g[V];
        Wide<T>::unpack(nw[c], g);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float& e = xs[r * p.K + c * V + j];
          e = Wide<T>::round(e * inv * g[j]);   // the norm's result has the type of x
        }
      }
    }
  }
  __syncthreads();
  float acc[WR][R];
#pragma unroll
  for (int i = 0; i < WR; ++i)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[i][r] = 0.f;
  for (int c = lane; c < chunks; c += 32) {
    float wv[WR][V];
#pragma unroll
    for (int i = 0; i < WR; ++i) Wide<T>::unpack(q[i], wv[i]);
    if (c + 32 < chunks) {
#pragma unroll
      for (int i = 0; i < WR; ++i) q[i] = wrow[i][c + 32];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int j = 0; j < V; j += 4) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + r * p.K + c * V + j);
#pragma unroll
        for (int i = 0; i < WR; ++i) {
          acc[i][r] = fmaf(wv[i][j], xv.x, acc[i][r]);
          acc[i][r] = fmaf(wv[i][j + 1], xv.y, acc[i][r]);
          acc[i][r] = fmaf(wv[i][j + 2], xv.z, acc[i][r]);
          acc[i][r] = fmaf(wv[i][j + 3], xv.w, acc[i][r]);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < WR; ++i)
#pragma unroll
    for (int r = 0; r < R; ++r) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[i][r] += __shfl_xor_sync(0xffffffffu, acc[i][r], o);
      if (lane == i * R + r && n0 + i < p.N && r < p.rows)
        reinterpret_cast<T*>(p.y)[(int64_t)r * p.N + n0 + i] = Wide<T>::cast(acc[i][r]);
    }
}

template <typename T, int R, int WR>
static int launch_token(const TokenLinearParams& p, cudaStream_t st) {
  const size_t smem = (size_t)R * p.K * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(castle_token_linear_kernel<T, R, WR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTokenSmem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_token_linear attribute");
  }
  constexpr int per_cta = kTokenThreads / 32 * WR;
  castle_token_linear_kernel<T, R, WR><<<(p.N + per_cta - 1) / per_cta, kTokenThreads, smem, st>>>(p);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_token_linear launch");
}
template <typename T, int R>
static int launch_token_r(const TokenLinearParams& p, cudaStream_t st) {
  // one row of w per warp until that fills the SMs (its latency is the time), four from there on (loads in flight)
  return p.N < 148 * 16 ? launch_token<T, R, 1>(p, st) : launch_token<T, R, 4>(p, st);
}
template <typename T>
static int launch_token_t(const TokenLinearParams& p, cudaStream_t st) {
  return p.rows == 1 ? launch_token_r<T, 1>(p, st) : p.rows == 2 ? launch_token_r<T, 2>(p, st)
         : p.rows <= 4 ? launch_token_r<T, 4>(p, st) : launch_token_r<T, 8>(p, st);
}

static int token_rows(int rows) { return rows <= 2 ? rows : rows <= 4 ? 4 : 8; }

}  // namespace castle

using namespace castle;

extern "C" int castle_token_linear_fits(int32_t dtype, int32_t rows, int32_t in_features) {
  return dtype >= CASTLE_BF16 && dtype <= CASTLE_F32 && rows >= 1 && rows <= 8 && in_features > 0 && in_features % 8 == 0 &&
         (int64_t)token_rows(rows) * in_features * (int64_t)sizeof(float) <= kTokenSmem;
}

extern "C" int castle_token_linear(int32_t dtype, int32_t rows, int32_t in_features, int32_t out_features, const void* x,
                                   int64_t row_stride, const void* norm_weight, float eps, const void* weight, void* y,
                                   void* stream) {
  if (!castle_token_linear_fits(dtype, rows, in_features) || out_features <= 0)
    return reject("castle_token_linear: %d rows of %d -> %d not supported (1 to 8 rows, in_features a multiple of 8)", rows, in_features, out_features);
  if (!x || !weight || !y) return reject("castle_token_linear: null tensor");
  if (((uintptr_t)x | (uintptr_t)weight | (uintptr_t)norm_weight) % 16 || row_stride * elem_size(dtype) % 16)
    return reject("castle_token_linear: pointers and the row stride must be 16-byte aligned");
  const TokenLinearParams p{x, norm_weight, weight, y, rows, in_features, out_features, row_stride, eps};
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == CASTLE_BF16) return launch_token_t<__nv_bfloat16>(p, st);
  if (dtype == CASTLE_F16) return launch_token_t<__half>(p, st);
  return launch_token_t<float>(p, st);
}
