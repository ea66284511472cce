// Small matrix products: the projections around the core, forward and backward, of calls that are short enough for the host
// to be the bound.  A library product costs the host 8 to 10 us (its heuristics, handles and checks) where a launch costs 3;
// a short prompt has two of them and a small training step six.  Large products stay with the library (see small_product in
// host.cpp, where the line lies and what both sides measured).
//
//   layout 0:  C[m,n] = A[m,k] B[n,k]^T      y = x w^T
//   layout 1:  C[m,n] = A[m,k] B[k,n]        dx = dy w
//   layout 2:  C[m,n] = A[k,m]^T B[k,n]      dw = dy^T x
//
// What bounds them on the GPU is the chain of one tile (fill, a handful of chunks, drain), not a rate: 197 x 512 -> 3072 in bf16
// takes 4.9 us.  With own products a prompt of 197 positions went from 60 to 49 us, a training step of 2 x 256 in fp32 from 187
// to 155.
//
// 16-bit types: one CTA per 128 x BN tile, tcgen05 products on chunks of 128 of k that TMA brings in, fp32 accumulators in
// tensor memory; every layout reads its operands as they lie (down their columns where k is the slow index).  fp32: FMA, see below.
#include "common.cuh"
#include "sm100.cuh"

namespace castle {

constexpr int kLinThreads = 128, kLinStages = 3, kLinChunk = 128;
constexpr uint32_t kLinPanel = 128 * 128;   // [128 rows][64 x 16 bit]

struct LinearParams {
  void* c;
  int m, n, k;
  int64_t ldc;
  int32_t* status;
};

template <int BN> constexpr uint32_t kLinStage = 2 * kLinPanel + (BN == 128 ? 2 : 1) * kLinPanel;   // BN = 64, layout 0: two panels of 64 rows
template <int BN> constexpr size_t kLinSmem = kLinStages * kLinStage<BN> + 1024;

template <typename T, int LAYOUT, int BN>
__global__ void __launch_bounds__(kLinThreads) castle_linear_kernel(const LinearParams p, const __grid_constant__ CUtensorMap m_a,
                                                                    const __grid_constant__ CUtensorMap m_b) {
  constexpr int FMT = Elem<T>::fmt;
  constexpr bool A_MN = LAYOUT == 2, B_MN = LAYOUT != 0;
  constexpr uint32_t IDESC = make_idesc(128, BN, FMT, A_MN, B_MN, false);
  constexpr uint32_t B_PANEL = !B_MN && BN == 64 ? kLinPanel / 2 : kLinPanel;   // layout 0: BN rows of 64 k each
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t bar_full[kLinStages], bar_free[kLinStages], bar_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * 128;
  const int chunks = (p.k + kLinChunk - 1) / kLinChunk;
  if (tid == 0) {
    for (int s = 0; s < kLinStages; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_free[s], 1); }
    mbar_init(&bar_done, 1);
    mbar_fence_init();
    abort_flag = 0;
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, BN); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s, trow = tmem + ((uint32_t)(warp * 32) << 16);
  volatile int* abortp = &abort_flag;
  if (tid == 0) {
    auto load = [&](int c) {   // chunk c: two panels of A, of B as many as it has (k or n beyond the matrix reads as zero)
      uint8_t* a = smem + (c % kLinStages) * kLinStage<BN>;
      uint8_t* b = a + 2 * kLinPanel;
      uint64_t* bar = &bar_full[c % kLinStages];
      mbar_expect_tx(bar, kLinStage<BN>);
#pragma unroll
      for (int pn = 0; pn < 2; ++pn) {
        if (A_MN) tma_load_4d(a + pn * kLinPanel, &m_a, bar, m0 + pn * 64, c * kLinChunk, 0, 0);
        else tma_load_4d(a + pn * kLinPanel, &m_a, bar, c * kLinChunk + pn * 64, m0, 0, 0);
        if (!B_MN) tma_load_4d(b + pn * B_PANEL, &m_b, bar, c * kLinChunk + pn * 64, n0, 0, 0);
        else if (pn * 64 < BN) tma_load_4d(b + pn * kLinPanel, &m_b, bar, n0 + pn * 64, c * kLinChunk, 0, 0);
      }
    };
    for (int c = 0; c < kLinStages && c < chunks; ++c) load(c);
    for (int c = 0; c < chunks; ++c) {
      const int s = c % kLinStages;
      mbar_wait(&bar_full[s], (uint32_t)(c / kLinStages) & 1u, abortp);
      tc_fence_after();
      const uint32_t a = smem_u32(smem) + s * kLinStage<BN>, b = a + 2 * kLinPanel;
      if constexpr (LAYOUT == 0) {
        const uint64_t da = desc_kmajor(a), db = desc_kmajor(b);
#pragma unroll
        for (int q = 0; q < 8; ++q)
          mma_ss(tmem, da + (uint64_t)(((q >> 2) * kLinPanel + 32 * (q & 3)) >> 4), db + (uint64_t)(((q >> 2) * B_PANEL + 32 * (q & 3)) >> 4), IDESC,
                 c > 0 || q > 0);
      } else if constexpr (LAYOUT == 1) {
        gemm_km_t<8>(tmem, a, b, IDESC, c > 0);
      } else {
        gemm_mm_t<8>(tmem, a, b, IDESC, c > 0);
      }
      mma_commit(c + 1 == chunks ? &bar_done : &bar_free[s]);
      if (c > 0 && c - 1 + kLinStages < chunks) {   // the chunk before has been read: its stage is filled again
        mbar_wait(&bar_free[(c - 1) % kLinStages], (uint32_t)((c - 1) / kLinStages) & 1u, abortp);
        load(c - 1 + kLinStages);
      }
    }
  }
  __syncwarp();
  mbar_wait(&bar_done, 0, abortp);
  tc_fence_after();
  // ---- through shared memory, so that eight lanes store a row's 128 bytes
  uint8_t* out = smem + warp * 32 * 128;   // per warp: 32 rows of a panel
#pragma unroll
  for (int c = 0; c < BN / 32; ++c) {
    float v[32];
    tmem_ld32(trow + c * 32, v);
    tmem_ld_wait();
    store_row32<T>(out, kLinPanel, lane, c * 32, v);
  }
  __syncwarp();
  T* dst = reinterpret_cast<T*>(p.c);
#pragma unroll
  for (int pn = 0; pn < BN / 64; ++pn) {
    const int col = n0 + pn * 64 + (lane & 7) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int r = j * 4 + (lane >> 3), row = m0 + warp * 32 + r;
      if (row < p.m && col < p.n)
        *reinterpret_cast<uint4*>(dst + (int64_t)row * p.ldc + col) = *reinterpret_cast<const uint4*>(out + pn * kLinPanel + swz_off(r, lane & 7));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, BN);
  if (tid == 0 && abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

// fp32: a CTA of eight groups of 64 threads owns a 32 x 32 tile; each group sums an eighth of k (a thread 4 x 4 values), the sums
// meet in shared memory in the order of the groups.  Small products have few tiles, and one long chain over k is their time
// (512 x 768 -> 128: 10.2 us, with four groups on 32 x 64 tiles 17.1, the library 14.4).
constexpr int kF32Groups = 8, kF32Group = 64, kF32Tile = 32, kF32K = 16, kF32Ld = kF32Tile + 4;
constexpr int kF32Stage = 2 * kF32K * kF32Ld, kF32Smem = kF32Groups * 2 * kF32Stage * (int)sizeof(float);
struct LinearF32Params {
  const float *a, *b;
  float* c;
  int m, n, k;
  int64_t lda, ldb, ldc;
};
template <int LAYOUT>
__global__ void __launch_bounds__(kF32Groups * kF32Group) castle_linear_f32_kernel(const LinearF32Params p) {
  constexpr bool A_MN = LAYOUT == 2, B_MN = LAYOUT != 0;
  extern __shared__ __align__(16) float f32_smem[];   // [group][2][A then B: k][32 + 4]
  const int tid = threadIdx.x % kF32Group, grp = threadIdx.x / kF32Group;
  const int n0 = blockIdx.x * kF32Tile, m0 = blockIdx.y * kF32Tile;
  const int share = ((p.k + kF32Groups - 1) / kF32Groups + 3) / 4 * 4, k_begin = grp * share, k_end = min(p.k, k_begin + share);
  const int steps = max(0, (k_end - k_begin + kF32K - 1) / kF32K);
  // a chunk of an operand is 32 x 16 values: two float4 a thread, along k or along the tile (all extents are multiples of four)
  auto load = [&](const float* src, int64_t ld, bool mn, int o0, int end, int k0, int i) {
    const int e = tid + kF32Group * i, o = o0 + (mn ? (e & 7) * 4 : e >> 2), k = k0 + (mn ? e >> 3 : (e & 3) * 4);
    return o < end && k < k_end ? *reinterpret_cast<const float4*>(src + (mn ? k * ld + o : o * ld + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  auto put = [&](float* s, bool mn, const float4& v, int i) {
    const int e = tid + kF32Group * i;
    if (mn) {
      *reinterpret_cast<float4*>(s + (e >> 3) * kF32Ld + (e & 7) * 4) = v;
    } else {
      float* d = s + (e & 3) * 4 * kF32Ld + (e >> 2);
      d[0] = v.x; d[kF32Ld] = v.y; d[2 * kF32Ld] = v.z; d[3 * kF32Ld] = v.w;
    }
  };
  const int tx = tid & 7, ty = tid >> 3;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float4 a[2][2], b[2][2];   // two chunks on their way
  auto fetch = [&](int q, int s) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      a[q][i] = load(p.a, p.lda, A_MN, m0, p.m, k_begin + s * kF32K, i);
      b[q][i] = load(p.b, p.ldb, B_MN, n0, p.n, k_begin + s * kF32K, i);
    }
  };
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (q < steps) fetch(q, q);
  for (int s0 = 0; s0 < steps; s0 += 2) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int s = s0 + q;
      if (s >= steps) break;
      float* cur = f32_smem + (grp * 2 + q) * kF32Stage;
#pragma unroll
      for (int i = 0; i < 2; ++i) { put(cur, A_MN, a[q][i], i); put(cur + kF32K * kF32Ld, B_MN, b[q][i], i); }
      if (s + 2 < steps) fetch(q, s + 2);
      asm volatile("bar.sync %0, 64;" ::"r"(1 + grp) : "memory");   // (this buffer's last readers have passed the other buffer's barrier)
#pragma unroll
      for (int k = 0; k < kF32K; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(cur + k * kF32Ld + ty * 4);
        const float4 y = *reinterpret_cast<const float4*>(cur + (kF32K + k) * kF32Ld + tx * 4);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xs[i], ys[j], acc[i][j]);
      }
    }
  }
  __syncthreads();
  float* red = f32_smem + grp * kF32Tile * kF32Tile;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(red + (ty * 4 + i) * kF32Tile + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
  const int row = threadIdx.x >> 4, col = (threadIdx.x & 15) * 2;   // two values a thread
  float2 sum = *reinterpret_cast<const float2*>(f32_smem + row * kF32Tile + col);
#pragma unroll
  for (int g = 1; g < kF32Groups; ++g) {
    const float2 v = *reinterpret_cast<const float2*>(f32_smem + (g * kF32Tile + row) * kF32Tile + col);
    sum.x += v.x; sum.y += v.y;
  }
  if (m0 + row < p.m && n0 + col < p.n) *reinterpret_cast<float2*>(p.c + (int64_t)(m0 + row) * p.ldc + n0 + col) = sum;
}

// Tensor map over a row-major 16-bit matrix: box of 64 columns x `box_rows`.
static int make_tmap_matrix(CUtensorMap* m, const void* base, int dtype, int64_t rows, int64_t cols, int64_t ld, int box_rows, const char* name) {
  const castle_tensor_t t{const_cast<void*>(base), rows * ld, rows * ld, ld};
  if (rows > 2147483647LL || cols > 2147483647LL) return reject("%s: too large", name);
  return make_tmap_16bit(m, &t, dtype, 1, 1, (int)rows, (int)cols, box_rows, name);
}

template <typename T, int LAYOUT, int BN>
static int launch_linear(const LinearParams& p, const void* a, int64_t lda, const void* b, int64_t ldb, int dtype, cudaStream_t st) {
  CUtensorMap ma, mb;
  int rc = LAYOUT == 2 ? make_tmap_matrix(&ma, a, dtype, p.k, p.m, lda, 128, "a") : make_tmap_matrix(&ma, a, dtype, p.m, p.k, lda, 128, "a");
  if (rc) return rc;
  rc = LAYOUT == 0 ? make_tmap_matrix(&mb, b, dtype, p.n, p.k, ldb, BN, "b") : make_tmap_matrix(&mb, b, dtype, p.k, p.n, ldb, 128, "b");
  if (rc) return rc;
  cudaError_t e = cudaFuncSetAttribute(castle_linear_kernel<T, LAYOUT, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLinSmem<BN>);
  if (e != cudaSuccess) return cuda_fail(e, "castle_linear attribute");
  e = launch_kernel(castle_linear_kernel<T, LAYOUT, BN>, dim3((p.n + BN - 1) / BN, (p.m + 127) / 128), kLinThreads, kLinSmem<BN>, st, false, p, ma, mb);
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_linear launch");
}
template <typename T>
static int launch_linear_t(const LinearParams& p, int layout, const void* a, int64_t lda, const void* b, int64_t ldb, int dtype, cudaStream_t st) {
  // 64 columns a tile while that leaves SMs idle
  const bool narrow = (int64_t)((p.n + 127) / 128) * ((p.m + 127) / 128) < 148;
  switch (layout) {
    case 0: return narrow ? launch_linear<T, 0, 64>(p, a, lda, b, ldb, dtype, st) : launch_linear<T, 0, 128>(p, a, lda, b, ldb, dtype, st);
    case 1: return narrow ? launch_linear<T, 1, 64>(p, a, lda, b, ldb, dtype, st) : launch_linear<T, 1, 128>(p, a, lda, b, ldb, dtype, st);
    default: return narrow ? launch_linear<T, 2, 64>(p, a, lda, b, ldb, dtype, st) : launch_linear<T, 2, 128>(p, a, lda, b, ldb, dtype, st);
  }
}

}  // namespace castle

using namespace castle;

extern "C" int castle_linear(int32_t dtype, int32_t layout, int32_t m, int32_t n, int32_t k, const void* a, int64_t lda, const void* b,
                             int64_t ldb, void* c, int64_t ldc, int32_t* status, void* stream) {
  if (dtype < CASTLE_BF16 || dtype > CASTLE_F32) return reject("castle_linear: unknown dtype %d", dtype);
  if (layout < 0 || layout > 2) return reject("castle_linear: unknown layout %d", layout);
  if (m <= 0 || n <= 0 || k <= 0) return reject("castle_linear: empty product");
  if (!a || !b || !c || !status) return reject("castle_linear: null tensor");
  const int es = elem_size(dtype), unit = 16 / es;
  if (n % unit || (layout == 2 ? m : k) % unit)
    return reject("castle_linear: n, and k (m in layout 2) must be multiples of %d", unit);
  if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) % 16 || lda * es % 16 || ldb * es % 16 || ldc * es % 16)
    return reject("castle_linear: pointers and row strides must be 16-byte aligned");
  if (lda < (layout == 2 ? m : k) || ldb < (layout == 0 ? k : n) || ldc < n) return reject("castle_linear: a row stride is shorter than its row");
  if ((m + 31) / 32 > 65535) return reject("castle_linear: too many rows");
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == CASTLE_F32) {
    const LinearF32Params p{(const float*)a, (const float*)b, (float*)c, m, n, k, lda, ldb, ldc};
    const dim3 grid((n + kF32Tile - 1) / kF32Tile, (m + kF32Tile - 1) / kF32Tile);
    auto kernel = layout == 0 ? castle_linear_f32_kernel<0> : layout == 1 ? castle_linear_f32_kernel<1> : castle_linear_f32_kernel<2>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kF32Smem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_linear attribute");
    e = launch_kernel(kernel, grid, kF32Groups * kF32Group, kF32Smem, st, false, p);
    return e == cudaSuccess ? 0 : cuda_fail(e, "castle_linear launch");
  }
  const LinearParams p{c, m, n, k, ldc, status};
  return dtype == CASTLE_BF16 ? launch_linear_t<__nv_bfloat16>(p, layout, a, lda, b, ldb, dtype, st)
                              : launch_linear_t<__half>(p, layout, a, lda, b, ldb, dtype, st);
}
