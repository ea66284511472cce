// y = norm(x) @ w^T for the handful of rows a cached single-token step projects (one row per sequence).
//
// At this size the product is a stream over the weights, and what a library call costs is its host side: one RMSNorm
// and two linear calls took 30 us of the 36 us a bf16 token's layer took on the host, for 9 us of kernels.  Here the
// norm is folded into the projection (every CTA computes it from x, which it needs whole anyway) and a call is one
// launch.  A warp owns WR rows of w and streams them with 16-byte loads; x sits in shared memory as fp32; all sums are
// fp32.  At 1 x 512 -> 3072 -> 512 bf16 the kernels take 2.8 and 2.3 us where the library calls took 2.7 + 3.8 and 3.0.
#include "common.cuh"
#include "decode_row.cuh"
#include "vec.cuh"

namespace castle {

constexpr int kTokenThreads = 128;
constexpr int kTokenSmem = 96 * 1024;   // x as fp32

struct TokenLinearParams {
  const void *x, *norm, *w;
  void* y;
  int rows, K, N;
  int64_t ldx;
  float eps;
  bool overlap;   // launched before the kernel that writes x has ended
};

// R = rows of x (padded up to 1, 2, 4 or 8), WR = rows of w per warp.
template <typename T, int R, int WR>
__global__ void __launch_bounds__(kTokenThreads) castle_token_linear_kernel(const TokenLinearParams p) {
  constexpr int V = Vec<T>::N, NW = kTokenThreads / 32;
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
  overlap_next();
  overlap_wait();   // x may come from the launch before
  float ss[R];
#pragma unroll
  for (int r = 0; r < R; ++r) ss[r] = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + (int64_t)min(r, p.rows - 1) * p.ldx);
    for (int c = threadIdx.x; c < chunks; c += kTokenThreads) {
      float v[V];
      Vec<T>::unpack(src[c], v);
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
        Vec<T>::unpack(nw[c], g);
#pragma unroll
        for (int j = 0; j < V; ++j) {
          float& e = xs[r * p.K + c * V + j];
          e = round_to<T>(e * inv * g[j]);   // the norm's result has the type of x
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
    for (int i = 0; i < WR; ++i) Vec<T>::unpack(q[i], wv[i]);
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
      if (lane == i * R + r && n0 + i < p.N && r < p.rows) {
        T* y = reinterpret_cast<T*>(p.y) + (int64_t)r * p.N + n0 + i;
        if constexpr (sizeof(T) == 4) *y = acc[i][r];
        else *y = Elem<T>::from_f(acc[i][r]);
      }
    }
}

// Three to eight rows of a 16-bit type: a matrix product with mma.sync, the weights as the 16 x 16 operand and the tokens as
// its 8 columns, which keeps it a stream over the weights (with fp32 arithmetic, x from shared memory is read R times per
// weight: 33 us for 8 x 2176 -> 13056, here 14.7, weights from memory).  A CTA stages the
// normalised x once and walks `groups` groups of 16 weight rows; its warps are KS slices of K times 8 / KS groups at a
// time, so that narrow outputs fill the SMs too.  A lane's 16-byte load of a weight row holds eight adjacent k; both
// operands use the same permutation of k inside a block of 32 (lane t of a quad: k = 8t .. 8t + 7), so the loads need no
// shuffles.
struct TokenMmaParams {
  TokenLinearParams l;
  int ks, groups;   // K slices; groups of 16 weight rows per CTA
};
constexpr int kTokenMmaThreads = 256;

template <typename T> __device__ __forceinline__ void mma_16x8x16(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  if constexpr (Elem<T>::fmt == 1)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <typename T>
__global__ void __launch_bounds__(kTokenMmaThreads) castle_token_mma_kernel(const TokenMmaParams q) {
  const TokenLinearParams& p = q.l;
  constexpr int R = 8;
  extern __shared__ __align__(16) uint8_t raw[];
  const int kp = (p.K + 31) / 32 * 32, ldx = kp + 8;        // K padded with zeros; 16 bytes of row padding against bank conflicts
  T* xs = reinterpret_cast<T*>(raw);                         // [R][ldx]
  float* red = reinterpret_cast<float*>(raw + (size_t)R * ldx * sizeof(T));   // [8 warps][16][R] where K is sliced
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  overlap_next();
  overlap_wait();   // x may come from the launch before
  // ---- x, normalised, into shared memory: a warp per row
  for (int r = warp; r < R; r += kTokenMmaThreads / 32) {
    const T* src = reinterpret_cast<const T*>(p.x) + (int64_t)min(r, p.rows - 1) * p.ldx;
    float inv = 1.f;
    if (p.norm && r < p.rows) {
      float ss = 0.f;
#pragma unroll 8
      for (int c = lane * 8; c < p.K; c += 256) {
        float v[8];
        load8<T>(src + c, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) ss = fmaf(v[j], v[j], ss);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      inv = rsqrtf(ss / (float)p.K + p.eps);
    }
#pragma unroll 4
    for (int c = lane * 8; c < kp; c += 256) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < p.rows && c < p.K) {
        v = *reinterpret_cast<const uint4*>(src + c);
        if (p.norm) {
          float f[8], g[8];
          load8<T>(src + c, f);
          load8<T>(reinterpret_cast<const T*>(p.norm) + c, g);
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = f[j] * inv * g[j];
          v = make_uint4(Elem<T>::pack2(f[0], f[1]), Elem<T>::pack2(f[2], f[3]), Elem<T>::pack2(f[4], f[5]), Elem<T>::pack2(f[6], f[7]));
        }
      }
      *reinterpret_cast<uint4*>(xs + (size_t)r * ldx + c) = v;
    }
  }
  __syncthreads();
  const int side = 8 / q.ks;                      // groups worked on at a time
  const int slice = warp % q.ks, col = warp / q.ks;
  const int g = lane >> 2, t = lane & 3;          // weight row (and token) inside a tile, k quarter
  const int blocks = kp / 32, b_begin = blocks * slice / q.ks, b_end = blocks * (slice + 1) / q.ks;
  for (int i = 0; i < q.groups; i += side) {
    const int n0 = (blockIdx.x * q.groups + i + col) * 16;
    const bool mine = i + col < q.groups && n0 < p.N;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    if (mine) {
      const T* w0 = reinterpret_cast<const T*>(p.w) + (int64_t)min(n0 + g, p.N - 1) * p.K + t * 8;
      const T* w1 = reinterpret_cast<const T*>(p.w) + (int64_t)min(n0 + g + 8, p.N - 1) * p.K + t * 8;
      constexpr int PF = 4;                       // blocks of 32 k in flight
      uint4 a0[PF], a1[PF];
      auto fetch = [&](int s, int blk) {
        const bool in = blk < b_end && blk * 32 + t * 8 < p.K;
        a0[s] = in ? *reinterpret_cast<const uint4*>(w0 + blk * 32) : make_uint4(0, 0, 0, 0);
        a1[s] = in ? *reinterpret_cast<const uint4*>(w1 + blk * 32) : make_uint4(0, 0, 0, 0);
      };
#pragma unroll
      for (int s = 0; s < PF; ++s) fetch(s, b_begin + s);
      for (int blk = b_begin; blk < b_end; blk += PF) {
#pragma unroll
        for (int s = 0; s < PF; ++s) {
          if (blk + s >= b_end) break;
          const uint4 u = a0[s], v = a1[s];
          fetch(s, blk + s + PF);
          const uint32_t lo[4] = {u.x, v.x, u.y, v.y}, hi[4] = {u.z, v.z, u.w, v.w};
          const uint4 b = *reinterpret_cast<const uint4*>(xs + (size_t)g * ldx + (blk + s) * 32 + t * 8);
          mma_16x8x16<T>(acc, lo, b.x, b.y);
          mma_16x8x16<T>(acc, hi, b.z, b.w);
        }
      }
    }
    // acc: rows n0 + g (0, 1) and n0 + g + 8 (2, 3), tokens 2t, 2t + 1
    if (q.ks > 1) {
      float* mine_red = red + (size_t)warp * 16 * R;
      *reinterpret_cast<float2*>(mine_red + g * R + 2 * t) = make_float2(acc[0], acc[1]);
      *reinterpret_cast<float2*>(mine_red + (g + 8) * R + 2 * t) = make_float2(acc[2], acc[3]);
      __syncthreads();
      for (int e = threadIdx.x; e < side * 16 * R; e += kTokenMmaThreads) {
        const int c = e / (16 * R), rest = e % (16 * R), tok = rest / 16, row = rest % 16;
        const int n = (blockIdx.x * q.groups + i + c) * 16 + row;
        if (i + c < q.groups && n < p.N && tok < p.rows) {
          float sum = 0.f;
          for (int k = 0; k < q.ks; ++k) sum += red[(size_t)(c * q.ks + k) * 16 * R + row * R + tok];
          reinterpret_cast<T*>(p.y)[(int64_t)tok * p.N + n] = Elem<T>::from_f(sum);
        }
      }
      __syncthreads();
    } else if (mine) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int row = n0 + g + (j >> 1) * 8, tok = 2 * t + (j & 1);
        if (row < p.N && tok < p.rows) reinterpret_cast<T*>(p.y)[(int64_t)tok * p.N + row] = Elem<T>::from_f(acc[j]);
      }
    }
  }
}

static size_t token_mma_smem(int K) { return (size_t)8 * ((K + 31) / 32 * 32 + 8) * 2 + (size_t)8 * 16 * 8 * sizeof(float); }
constexpr size_t kTokenMmaSmem = 200 * 1024;

template <typename T>
static int launch_token_mma(const TokenLinearParams& p, cudaStream_t st) {
  const size_t smem = token_mma_smem(p.K);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(castle_token_mma_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTokenMmaSmem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_token_linear attribute");
  }
  // the CTAs of one wave (three of 256 threads per SM, fewer where x is large); K is sliced as far as the groups of 16 rows
  // leave warps without one
  TokenMmaParams q{p, 1, 1};
  const int total = (p.N + 15) / 16, ctas = 148 * (smem > 110 * 1024 ? 1 : smem > 70 * 1024 ? 2 : 3);
  q.groups = (total + ctas - 1) / ctas;
  while (q.ks < 8 && q.groups * q.ks * 2 <= 8) q.ks *= 2;
  const int side = 8 / q.ks;
  q.groups = (q.groups + side - 1) / side * side;
  cudaError_t e = launch_kernel(castle_token_mma_kernel<T>, dim3((total + q.groups - 1) / q.groups), kTokenMmaThreads, smem, st, p.overlap, q);
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_token_linear launch");
}

template <typename T, int R, int WR>
static int launch_token(const TokenLinearParams& p, cudaStream_t st) {
  const size_t smem = (size_t)R * p.K * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(castle_token_linear_kernel<T, R, WR>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTokenSmem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_token_linear attribute");
  }
  constexpr int per_cta = kTokenThreads / 32 * WR;
  cudaError_t e = launch_kernel(castle_token_linear_kernel<T, R, WR>, dim3((p.N + per_cta - 1) / per_cta), kTokenThreads, smem, st, p.overlap, p);
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_token_linear launch");
}
template <typename T, int R>
static int launch_token_r(const TokenLinearParams& p, cudaStream_t st) {
  // one row of w per warp until that fills the SMs (its latency is the time), four from there on (loads in flight)
  return p.N < 148 * 16 ? launch_token<T, R, 1>(p, st) : launch_token<T, R, 4>(p, st);
}
template <typename T>
static int launch_token_t(const TokenLinearParams& p, cudaStream_t st) {
  if constexpr (sizeof(T) == 2) {
    if (p.rows > 2) return launch_token_mma<T>(p, st);
  }
  return p.rows == 1 ? launch_token_r<T, 1>(p, st) : p.rows == 2 ? launch_token_r<T, 2>(p, st)
         : p.rows <= 4 ? launch_token_r<T, 4>(p, st) : launch_token_r<T, 8>(p, st);
}

static int token_rows(int rows) { return rows <= 2 ? rows : rows <= 4 ? 4 : 8; }

}  // namespace castle

using namespace castle;

extern "C" int castle_token_linear_fits(int32_t dtype, int32_t rows, int32_t in_features) {
  if (dtype < CASTLE_BF16 || dtype > CASTLE_F32 || rows < 1 || in_features <= 0 || in_features % 8) return 0;
  if (dtype != CASTLE_F32 && rows > 2) return rows <= 8 && token_mma_smem(in_features) <= kTokenMmaSmem;
  return rows <= 8 && (int64_t)token_rows(rows) * in_features * (int64_t)sizeof(float) <= kTokenSmem;
}

extern "C" int castle_token_linear(int32_t dtype, int32_t rows, int32_t in_features, int32_t out_features, const void* x,
                                   int64_t row_stride, const void* norm_weight, float eps, const void* weight, void* y,
                                   int32_t overlap, void* stream) {
  if (!castle_token_linear_fits(dtype, rows, in_features) || out_features <= 0)
    return reject("castle_token_linear: %d rows of %d -> %d not supported (see castle_token_linear_fits)", rows, in_features, out_features);
  if (!x || !weight || !y) return reject("castle_token_linear: null tensor");
  if (((uintptr_t)x | (uintptr_t)weight | (uintptr_t)norm_weight) % 16 || row_stride * elem_size(dtype) % 16)
    return reject("castle_token_linear: pointers and the row stride must be 16-byte aligned");
  const TokenLinearParams p{x, norm_weight, weight, y, rows, in_features, out_features, row_stride, eps, overlap != 0};
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == CASTLE_BF16) return launch_token_t<__nv_bfloat16>(p, st);
  if (dtype == CASTLE_F16) return launch_token_t<__half>(p, st);
  return launch_token_t<float>(p, st);
}
