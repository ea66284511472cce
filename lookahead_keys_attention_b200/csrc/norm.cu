// RMSNorm of the module's input, forward and backward (the reference's `prenorm`).  At the language model's layer (16384
// rows of 512, bf16) the torch kernels took 21 us forward and 63 us backward, 45 of them for the weight's gradient; all
// of it is a few passes over 17 MB that stay in L2.
//
// Forward and dx: a warp per row, 16 bytes per lane and access, all sums fp32; the row is read twice (the second time
// from L1).  Weight gradient: a CTA owns 256 columns and a range of rows and leaves fp32 partials, which a second
// kernel adds in a fixed order, so the result is reproducible.  Both gradients of rows that fit a warp's registers: one kernel.
#include "common.cuh"
#include "vec.cuh"

namespace castle {

constexpr int kNormThreads = 256;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T>
__global__ void __launch_bounds__(kNormThreads) castle_rmsnorm_fwd_kernel(const T* __restrict__ x, const T* __restrict__ w, float eps,
                                                                          T* __restrict__ y, float* __restrict__ rstd, int64_t rows, int dim) {
  const int64_t r = (int64_t)blockIdx.x * (kNormThreads / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  const T* xr = x + r * dim;
  float ss = 0.f;
  for (int c = lane * 8; c < dim; c += 256) {
    float v[8];
    load8<T>(xr + c, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
  }
  const float inv = rsqrtf(warp_sum(ss) / (float)dim + eps);
  for (int c = lane * 8; c < dim; c += 256) {
    float v[8], g[8];
    load8<T>(xr + c, v);
    load8<T>(w + c, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = v[j] * inv * g[j];
    store8<T>(y + r * dim + c, v);
  }
  if (rstd && lane == 0) rstd[r] = inv;
}

// dx = rstd (dy w - x rstd^2 mean(dy w x))
template <typename T>
__global__ void __launch_bounds__(kNormThreads) castle_rmsnorm_dx_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ w,
                                                                         const float* __restrict__ rstd, T* __restrict__ dx, int64_t rows, int dim) {
  const int64_t r = (int64_t)blockIdx.x * (kNormThreads / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= rows) return;
  float dot = 0.f;
  for (int c = lane * 8; c < dim; c += 256) {
    float a[8], v[8], g[8];
    load8<T>(dy + r * dim + c, a);
    load8<T>(x + r * dim + c, v);
    load8<T>(w + c, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) dot = fmaf(a[j] * g[j], v[j], dot);
  }
  const float inv = rstd[r], k = warp_sum(dot) / (float)dim * inv * inv;
  for (int c = lane * 8; c < dim; c += 256) {
    float a[8], v[8], g[8];
    load8<T>(dy + r * dim + c, a);
    load8<T>(x + r * dim + c, v);
    load8<T>(w + c, g);
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = inv * (a[j] * g[j] - v[j] * k);
    store8<T>(dx + r * dim + c, a);
  }
}

// partial[blockIdx.y][column] = sum over the block's rows of dy x rstd: 32 lanes x 8 columns, 8 warps of rows
template <typename T>
__global__ void __launch_bounds__(kNormThreads) castle_rmsnorm_dw_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                         const float* __restrict__ rstd, float* __restrict__ partial,
                                                                         int64_t rows, int dim, int rows_per_block) {
  constexpr int NW = kNormThreads / 32;
  __shared__ float s[NW][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 256 + lane * 8;
  const int64_t r0 = (int64_t)blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  if (c < dim) {
#pragma unroll 4
    for (int64_t r = r0 + warp; r < r1; r += NW) {
      float a[8], v[8];
      load8<T>(dy + r * dim + c, a);
      load8<T>(x + r * dim + c, v);
      const float inv = rstd[r];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = fmaf(a[j] * inv, v[j], acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) s[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < dim) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < NW; ++k) t += s[k][threadIdx.x];
    partial[(int64_t)blockIdx.y * dim + col] = t;
  }
}

// Both gradients in one pass over dy and x: a warp takes every eighth row of its CTA's range, whole (C x 256 columns), the next
// row on its way meanwhile, and keeps its share of the weight's gradient in registers.  us of both gradients with the sum of the
// partials, replayed from a graph, a pass for each / so: 16384 x 512 bf16 15.6 / 10.2, fp32 30.9 / 16.6 (the bytes take 7.7 and 15.4 from
// memory), 50000 x 512 bf16 48.9 / 33.8, 200 x 512 bf16 5.7 / 4.7, 512 x 128 fp32 5.5 / 4.3.
template <typename T, int C>
__global__ void __launch_bounds__(kNormThreads, 2) castle_rmsnorm_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ w,
                                                                             const float* __restrict__ rstd, T* __restrict__ dx,
                                                                             float* __restrict__ partial, int64_t rows, int dim, int rows_per_block) {
  constexpr int NW = kNormThreads / 32;
  __shared__ float s[NW][C * 256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  auto column = [&](int q) { return q * 256 + lane * 8; };
  auto raw = [&](const T* p, int q) { return column(q) < dim ? *reinterpret_cast<const Raw8<T>*>(p + column(q)) : Raw8<T>{}; };
  Raw8<T> g[C], a[C], v[C];
  float acc[C][8], inv = 0.f;
#pragma unroll
  for (int q = 0; q < C; ++q) {
    g[q] = raw(w, q);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[q][j] = 0.f;
  }
  auto fetch = [&](int64_t r) {
#pragma unroll
    for (int q = 0; q < C; ++q) { a[q] = raw(dy + r * dim, q); v[q] = raw(x + r * dim, q); }
    inv = rstd[r];
  };
  if (r0 + warp < r1) fetch(r0 + warp);
  for (int64_t r = r0 + warp; r < r1; r += NW) {
    float fa[C][8], fv[C][8], dot = 0.f;
    const float iv = inv;
#pragma unroll
    for (int q = 0; q < C; ++q) {
      float fg[8];
      load8<T>(reinterpret_cast<const T*>(&a[q]), fa[q]);
      load8<T>(reinterpret_cast<const T*>(&v[q]), fv[q]);
      load8<T>(reinterpret_cast<const T*>(&g[q]), fg);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[q][j] = fmaf(fa[q][j] * iv, fv[q][j], acc[q][j]);
        dot = fmaf(fa[q][j] * fg[j], fv[q][j], dot);
      }
    }
    if (r + NW < r1) fetch(r + NW);
    const float k = warp_sum(dot) / (float)dim * iv * iv;
#pragma unroll
    for (int q = 0; q < C; ++q)
      if (column(q) < dim) {
        float fg[8];
        load8<T>(reinterpret_cast<const T*>(&g[q]), fg);
#pragma unroll
        for (int j = 0; j < 8; ++j) fa[q][j] = iv * fmaf(fa[q][j], fg[j], -(fv[q][j] * k));   // the smaller product is the rounded one
        store8<T>(dx + r * dim + column(q), fa[q]);
      }
  }
#pragma unroll
  for (int q = 0; q < C; ++q)
#pragma unroll
    for (int j = 0; j < 8; j += 4) *reinterpret_cast<float4*>(&s[warp][column(q) + j]) = make_float4(acc[q][j], acc[q][j + 1], acc[q][j + 2], acc[q][j + 3]);
  __syncthreads();
#pragma unroll
  for (int q = 0; q < C; ++q) {
    const int col = q * 256 + threadIdx.x;
    if (col < dim) {
      float t = 0.f;
#pragma unroll
      for (int k = 0; k < NW; ++k) t += s[k][col];
      partial[(int64_t)blockIdx.x * dim + col] = t;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(kNormThreads) castle_rmsnorm_dw_sum_kernel(const float* __restrict__ partial, T* __restrict__ dw, int parts, int dim) {
  // 32 columns per block, 8 threads of each adding every eighth part, in a fixed order
  __shared__ float s[8][32];
  const int col = blockIdx.x * 32 + (threadIdx.x & 31), k0 = threadIdx.x >> 5;
  float t = 0.f;
  overlap_wait();   // launched while the partials are being written
  if (col < dim) {
#pragma unroll 8
    for (int k = k0; k < parts; k += 8) t += partial[(int64_t)k * dim + col];
  }
  s[k0][threadIdx.x & 31] = t;
  __syncthreads();
  if (threadIdx.x < 32 && col < dim) {
#pragma unroll
    for (int k = 1; k < 8; ++k) t += s[k][threadIdx.x];
    if constexpr (sizeof(T) == 4) dw[col] = t;
    else dw[col] = Elem<T>::from_f(t);
  }
}

static int norm_parts(int64_t rows, int dim) {   // row ranges of the weight gradient: about four CTAs per SM, at least 32 rows each
  const int cols = (dim + 255) / 256;
  int64_t parts = 148 * 4 / cols, most = (rows + 31) / 32;
  if (parts > most) parts = most;
  return (int)(parts < 1 ? 1 : parts);
}

// One pass where both gradients are wanted and a row's values fit the registers of a warp (128 a thread): up to 512 columns (three and four
// times 256 spill).
template <typename T>
static bool norm_bwd_whole(int64_t rows, int dim, const T* dy, const T* x, const T* w, const float* rstd, T* dx, float* ws, int parts, cudaStream_t st) {
  const int per = (int)((rows + parts - 1) / parts);
  auto go = [&](auto kernel) { kernel<<<parts, kNormThreads, 0, st>>>(dy, x, w, rstd, dx, ws, rows, dim, per); return true; };
  if (dim <= 256) return go(castle_rmsnorm_bwd_kernel<T, 1>);
  if (dim <= 512) return go(castle_rmsnorm_bwd_kernel<T, 2>);
  return false;
}

template <typename T>
static cudaError_t norm_bwd(int64_t rows, int dim, const void* dy, const void* x, const void* w, const float* rstd, void* dx, void* dw,
                            float* ws, cudaStream_t st) {
  const int parts = norm_parts(rows, dim), per = (int)((rows + parts - 1) / parts);
  if (!dx || !dw || !norm_bwd_whole<T>(rows, dim, (const T*)dy, (const T*)x, (const T*)w, rstd, (T*)dx, ws, parts, st)) {
    if (dx) castle_rmsnorm_dx_kernel<T><<<(unsigned)((rows + 7) / 8), kNormThreads, 0, st>>>((const T*)dy, (const T*)x, (const T*)w, rstd, (T*)dx, rows, dim);
    if (dw) castle_rmsnorm_dw_kernel<T><<<dim3((dim + 255) / 256, parts), kNormThreads, 0, st>>>((const T*)dy, (const T*)x, rstd, ws, rows, dim, per);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && dw) e = launch_kernel(castle_rmsnorm_dw_sum_kernel<T>, dim3((dim + 31) / 32), kNormThreads, 0, st, true, (const float*)ws, (T*)dw, parts, dim);
  return e;
}

static int norm_check(const char* who, int32_t dtype, int64_t rows, int32_t dim) {
  if (dtype < CASTLE_BF16 || dtype > CASTLE_F32) return reject("%s: unknown dtype", who);
  if (rows <= 0 || rows > (int64_t)8 * 2147483647 || dim <= 0 || dim % 8) return reject("%s: rows %lld, dim %d not supported (dim a multiple of 8)", who, (long long)rows, dim);
  return 0;
}

}  // namespace castle

using namespace castle;

extern "C" int castle_rmsnorm_fwd(int32_t dtype, int64_t rows, int32_t dim, const void* x, const void* weight, float eps, void* y,
                                  float* rstd, void* stream) {
  if (int rc = norm_check("castle_rmsnorm_fwd", dtype, rows, dim)) return rc;
  if (!x || !weight || !y || ((uintptr_t)x | (uintptr_t)weight | (uintptr_t)y) % 16)
    return reject("castle_rmsnorm_fwd: x, weight and y must be 16-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned grid = (unsigned)((rows + 7) / 8);
  if (dtype == CASTLE_BF16)
    castle_rmsnorm_fwd_kernel<__nv_bfloat16><<<grid, kNormThreads, 0, st>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)weight, eps, (__nv_bfloat16*)y, rstd, rows, dim);
  else if (dtype == CASTLE_F16)
    castle_rmsnorm_fwd_kernel<__half><<<grid, kNormThreads, 0, st>>>((const __half*)x, (const __half*)weight, eps, (__half*)y, rstd, rows, dim);
  else
    castle_rmsnorm_fwd_kernel<float><<<grid, kNormThreads, 0, st>>>((const float*)x, (const float*)weight, eps, (float*)y, rstd, rows, dim);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_rmsnorm_fwd launch");
}

extern "C" size_t castle_rmsnorm_bwd_workspace_bytes(int64_t rows, int32_t dim) {
  return rows <= 0 || dim <= 0 ? 0 : (size_t)norm_parts(rows, dim) * dim * sizeof(float);
}

extern "C" int castle_rmsnorm_bwd(int32_t dtype, int64_t rows, int32_t dim, const void* dy, const void* x, const void* weight,
                                  const float* rstd, void* dx, void* dweight, void* workspace, size_t workspace_bytes, void* stream) {
  if (int rc = norm_check("castle_rmsnorm_bwd", dtype, rows, dim)) return rc;
  if (!dy || !x || !weight || !rstd || ((uintptr_t)dy | (uintptr_t)x | (uintptr_t)weight | (uintptr_t)dx) % 16)
    return reject("castle_rmsnorm_bwd: dy, x, weight and dx must be 16-byte aligned");
  if (dweight && (!workspace || workspace_bytes < castle_rmsnorm_bwd_workspace_bytes(rows, dim)))
    return reject("castle_rmsnorm_bwd: workspace too small");
  cudaStream_t st = (cudaStream_t)stream;
  const cudaError_t e = dtype == CASTLE_BF16 ? norm_bwd<__nv_bfloat16>(rows, dim, dy, x, weight, rstd, dx, dweight, (float*)workspace, st)
                        : dtype == CASTLE_F16 ? norm_bwd<__half>(rows, dim, dy, x, weight, rstd, dx, dweight, (float*)workspace, st)
                                              : norm_bwd<float>(rows, dim, dy, x, weight, rstd, dx, dweight, (float*)workspace, st);
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_rmsnorm_bwd launch");
}
