// CASTLE parallel forward for sm_100a.
//
// The reference evaluates Su = T @ A^T as an (N x N) x (N x N) product, O(N^3)
// per head.  Here each CTA owns one block K of 128 keys and walks the query
// blocks I = K, K+1, ... keeping the running lookahead state
//     W_K = sum_{J < I} A[K,J] @ Vu[J]          (128 x d, fp32, in tensor memory)
// so that
//     Su[I,K] = Qc[I] @ W_K^T + tril(T[I,I]) @ A[K,I]^T
// costs O(N^2 d) in total.  Per (I,K) step the CTA issues seven tcgen05 products
// (Z, W update, T, Su main, Su in-block term, Sc, P@Vc), all with fp32
// accumulators in TMEM and 16-bit operands in 128-byte-swizzled shared memory,
// either loaded by TMA (inputs) or written by the threads (sigmoid gate A,
// masked T, the 16-bit copy of W, soft-max numerators P).  A thread owns 32
// consecutive columns of one accumulator row; row maxima and sums of the four
// threads sharing a row meet in shared memory.
//
// The soft-max over keys crosses CTAs, so each step emits an un-normalised
// partial (row max, row sum, P@Vc) and a second kernel merges the partials of a
// query block.  After the last step W_K is exactly U[K], the lookahead keys the
// decode cache stores, and (unrounded) the state the backward starts from.
#include <algorithm>
#include "common.cuh"
#include "sm100.cuh"

namespace castle {

constexpr int kBlk = 128;                       // keys per CTA, queries per step
constexpr uint32_t kPanelBytes = kBlk * 128;    // [128 rows][64 x 16-bit]

struct FwdParams {
  int B, H, N, nblk;
  float scale;
  float* part_ml;   // [BH][ntiles][128][2]
  void* part_o;     // [BH][ntiles][D/8][128][8] in the operand type (un-normalised P@Vc of one tile): a thread that owns a
                    // row stores 16-byte chunks, and a warp's store of one chunk is 512 contiguous bytes
  float* lse;       // [BH][N]
  float* w_state;   // [BH][N][D] or null
  castle_tensor_t u_out;  // ptr may be null
  int u_dtype;
  castle_tensor_t out;
  int32_t* status;
  int store_caches;   // also copy the Qu[K], Kc[K], Vc[K] tiles into the decode caches (prefill hand-off)
  uint4* tm;          // masked T tiles, or null
#ifdef CASTLE_PHASE_TIMING
  long long* timing;
#endif
};

__host__ __device__ inline int64_t tri(int64_t i) { return i * (i + 1) / 2; }

constexpr int kFwdThreads = 512;

constexpr int kSplitMin = 8;   // shorter walks are not cut
// First step of part `seg` of a walk of `walk` query blocks cut in `nseg` parts of equal cost: a part pays c = 0.45 of a
// step for each state-only step before it, so with parts beginning at x_i, c x_i + x_{i+1} - x_i is the same for all i.
__device__ inline int walk_cut(int walk, int nseg, int seg) {
  float a = 1.f, n = 1.f;
  for (int i = 0; i < nseg; ++i) {
    n *= 0.55f;
    if (i < seg) a *= 0.55f;
  }
  return (int)((float)walk * (1.f - a) / (1.f - n) + 0.5f);
}

// Optional phase timing (debug builds only): thread 0 of CTA (0,0) stores clock64() at each phase
// boundary of its first steps into the soft-max partial buffer's tail, which the host dumps.
#ifdef CASTLE_PHASE_TIMING
#define PIPE_MARK(i) do { if ((tid & 31) == 0 && (tid == 0 || tid == 256) && blockIdx.x == 0 && blockIdx.y == 0 && I - I_begin < 16) p.timing[(I - I_begin) * 16 + (i)] = clock64(); } while (0)
#else
#define PIPE_MARK(i) do { } while (0)
#endif

// ---------------------------------------------------------------------------------------------
// Two-stage pipeline: the step (I,K) is cut into a lookahead stage, run by warps 0-7 (X), and a soft-max stage, run by
// warps 8-15 (Y), and Y works on block I while X is on block I+1.  The chain between consecutive query blocks is only
// the state update, so the two overlap: X forms Z and the gate and issues every product up to the scores; Y turns Su
// and Sc into P, issues P @ Vc and stores the partial.  One CTA per SM; a group has 256 threads, each with 64 values
// of a 128x128 tile.
//
// The masked T[I,I] = tril(Qc[I] @ Vu[I]^T) is the same for every key block, so where that pays (fwd_plan, from kTmBlocks query
// blocks on) a small kernel computes the tiles once (castle_fwd_t_kernel) and X's threads carry theirs from global memory to tensor
// memory; that takes a product, an elementwise pass and two hand-offs out of X's chain.  Elsewhere (TM = false) X forms T itself.
//
// Tensor memory: W | R1 | R2 | R3 (| Tm), D + 3 * 128 (+ 64) columns.
//   R1  Z; at dim_head 128 then the masked T as packed pairs (first operand of the Su correction)
//   R2  Su; at dim_head 128 then P @ Vc
//   R3  Sc (issued by Y, as soon as these columns are free again), then P as packed pairs; at dim_head 64 its upper half
//       then takes P @ Vc
//
// Shared memory: Qu, Kc, Vc of the key block and the 16-bit copy of W stay.  dim_head 64: two buffers each of Ku, Vu, Qc
// and the gate, filled a step ahead.  dim_head 128: one of Qc and two 32 KB slots whose roles alternate: in step I slot P
// holds Ku[I] and, once Z is done, the gate over it; slot Q holds Vu[I] and then, after the state update, Ku[I+1];
// Vu[I+1] goes over the gate when the scores are done.
template <int D> struct FwdPipe {
  static constexpr uint32_t OPB = D / 64 * kPanelBytes;
  static constexpr uint32_t kRed = 224 * 1024;                  // row max and row sum of the two column halves
  static constexpr uint32_t kBars = kRed + 4 * kBlk * sizeof(float);
  static constexpr uint32_t kSmem = kBars + 192;
};

__device__ __forceinline__ void sync_x() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
// The two warps of a group that share 32 rows (and their tensor-memory lanes).
__device__ __forceinline__ void sync_pair(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void sync_y() { asm volatile("bar.sync 2, 256;" ::: "memory"); }

// 32 values of a row as the state or the lookahead keys (fp32, bf16 or fp16)
__device__ __forceinline__ void store_u32(void* base, int dtype, int64_t off, const float* v) {
  if (dtype == CASTLE_F32) {
    float* dst = reinterpret_cast<float*>(base) + off;
#pragma unroll
    for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(dst + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  } else {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(base) + off);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t q[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        q[i] = dtype == CASTLE_BF16 ? Elem<__nv_bfloat16>::pack2(v[8 * j + 2 * i], v[8 * j + 2 * i + 1])
                                    : Elem<__half>::pack2(v[8 * j + 2 * i], v[8 * j + 2 * i + 1]);
      dst[j] = make_uint4(q[0], q[1], q[2], q[3]);
    }
  }
}

// A masked T tile in global memory: [16 chunks of 8 columns][128 rows] x 16 bytes, so that a warp's access is contiguous.
constexpr int64_t kTmTile = 16 * kBlk;   // in uint4
constexpr int kTmBlocks = 8;             // with fewer query blocks they do not pay (64 x 16 heads x 6 blocks 709 / 697 us); from here on there is room for them (so that the scratch is linear in the pairs)

// The forward's plan for a problem: parts per walk, whether the masked T tiles are computed once, up front, and the kernel.
struct FwdPlan { int nseg; bool ahead, persistent; };
static FwdPlan fwd_plan(int64_t pairs, int64_t nblk, int dim_head) {
  FwdPlan f;
  // Few pairs: the grid is one wave whose length is the walk of key block 0, while the mean walk is half as long or, with
  // idle SMs, still less.  `load` = steps per SM over the longest walk.  us uncut / 2 / 3 parts: 4 pairs x 16 blocks at
  // dim_head 128 74 / 60 / 52 (load 0.23), 4 x 12 44 / 37 / 34 (0.18), 8 x 12 44 / 37 / 40 (0.35), 4 x 32 100 / 78 / 88 (0.45), 16 x 11
  // 43 / 46 / 52 (0.65), 8 x 32 103 / 138 / 166 (0.89).
  const float load = (float)pairs * (float)(nblk + 1) * (0.5f / 148.f);
  f.nseg = nblk < kSplitMin || load >= 0.6f ? 1 : load >= 0.3f ? 2 : 3;
  // The tiles cost 4 us of their kernel's latency and 7.5 ns (dim_head 64) or 12.5 ns a tile through memory; a step that reads one
  // instead of computing it is 0.43 and 0.36 us shorter (a product less in the chain).  The steps that count are those of the
  // busiest SM: their mean, or the longest walk, of whose parts some have few steps with scores.  us of a forward with /
  // without the tiles, pairs x blocks: dim_head 64 128 x 8 155.0 / 157.8, 64 x 10 119.7 / 121.9, 128 x 11 261.7 / 269.6, 64 x 17 278 / 297, 16 x 17
  // 77.4 / 78.9, 8 x 24 88.6 / 96.7, 4 x 32 87.3 / 91.8, 48 x 8 70.0 / 69.2, 4 x 12 39.4 / 35.8, 2 x 24 63.7 / 61.8, 1 x 32 77.9 / 76.1; dim_head 128
  // 16 x 22 186 / 191, 64 x 24 772 / 797, 64 x 16 388.6 / 388.4, 16 x 16 106.9 / 106.5, 128 x 8 253.8 / 246.0, 64 x 11 209.7 / 207.4, 16 x 11 69.6 / 68.5.
  const float longest = (float)nblk * (f.nseg == 1 ? 1.f : f.nseg == 2 ? 0.7f : 0.25f);
  const float steps = std::max(longest, load * (float)nblk);
  const bool narrow = dim_head == 64;
  f.ahead = nblk >= kTmBlocks && steps * (narrow ? 0.43f : 0.36f) > 4.f + (narrow ? 0.0075f : 0.0125f) * (float)(pairs * nblk);
  // A CTA that takes one walk after the other covers their starts and ends, but its steps are some 4 % longer (it looks up
  // what comes next), so it is for short walks, and the longer they are the more of them there must be.  us of the kernel, walk after walk / a
  // CTA per walk, pairs x blocks: 128 x 8 124 / 145, 48 x 12 103 / 110, 128 x 13 286 / 314, 128 x 17 460 / 485, 128 x 20 622 / 648, 64 x 24
  // 442 / 447, 64 x 32 748 / 739; few: 32 x 8 45 / 47, 24 x 8 42 / 40, 40 x 12 102 / 104, 24 x 20 131 / 129, 20 x 24 158 / 148, 8 x 24 88 / 78.
  // Below eight blocks a CTA per walk is the better one while no SM's second walk outlasts the longest one: in one wave, or if the
  // second walk, which starts behind a first of nblk - 148 / pairs steps and is as short, ends in time (start and end of a walk count
  // 2.4 steps): 2 (nblk - 148 / pairs + 2.4) <= nblk + 2.4.  us of a forward, walk after walk / a CTA per walk: 37 x 1 11.3 / 10.9, 148 x 1
  // 13.2 / 12.7, 163 x 1 17.1 / 20.2, 71 x 2 16.4 / 16.0, 83 x 2 17.6 / 20.9, 42 x 3 20.2 / 19.6, 51 x 3 20.7 / 21.2, 41 x 4 24.2 / 23.1, 48 x 4 24.8 /
  // 25.4, 34 x 5 28.0 / 26.5, 45 x 5 30.0 / 32.1, 30 x 6 32.1 / 30.3, 39 x 6 33.9 / 35.7, 26 x 7 36.2 / 34.1, 34 x 7 38.5 / 39.7.
  // Not here: two CTAs an SM, a walk each, in half the tensor memory.  Some sizes would be 3 to 5 % faster than walk after walk (500 x 1
  // 27.2 / 28.6, 256 x 2 35.8 / 37.0, 256 x 3 62.6 / 65.5), the others of more than a wave are up to 20 % slower (2048 x 1 95.0 / 92.1, 500 x 3
  // 117 / 108, 256 x 7 270 / 224): not worth a third kernel.
  const bool few = pairs * nblk <= 148 || (float)pairs * ((float)nblk + 2.4f) <= 296.f;
  f.persistent = dim_head == 64 && f.nseg == 1 && nblk <= 24 && (nblk < kSplitMin ? !few : 9.f * load >= (float)nblk);
  return f;
}

// ---------------------------------------------------------------------------------------------
// The arithmetic of a step, as both kernels below run it.  A thread has 64 values of a 128 x 128 tile, columns cbase.. of one row;
// tensor-memory addresses have the lanes of its warp.

// Gate A = sigmoid(scale * Z), kept for j > k (rows k, columns j), into its swizzled tile
template <typename T>
__device__ __forceinline__ void gate_pass(uint32_t z, uint8_t* tile, int row, int cbase, float half_scale, bool diag) {
  float v[2][32];
  tmem_ld32(z + cbase, v[0]);
  tmem_ld32(z + cbase + 32, v[1]);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < 2; ++c) {
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float2 a = sigmoid2(make_float2(v[c][j], v[c][j + 1]), half_scale);
      v[c][j] = a.x; v[c][j + 1] = a.y;
    }
    if (diag) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[c][j] = (cbase + c * 32 + j > row) ? v[c][j] : 0.f;
    }
    store_row32<T>(tile, kPanelBytes, row, cbase + c * 32, v[c]);
  }
}

// The 16-bit copy of W; a group has half of the columns
template <typename T, int D>
__device__ __forceinline__ void state_copy(uint32_t w, uint8_t* tile, int row, int grp) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) {
    const int c0 = (grp * (D / 64) + c) * 32;
    float v[32];
    tmem_ld32(w + c0, v);
    tmem_ld_wait();
    store_row32<T>(tile, kPanelBytes, row, c0, v);
  }
}

// The final state of a walk, U[K], into the caller's tensors (either may be null)
template <int D>
__device__ __forceinline__ void state_out(const FwdParams& p, uint32_t w, int bh, int K, int row, int grp) {
  const int krow = K * kBlk + row;
#pragma unroll 1
  for (int c = 0; c < D / 64; ++c) {
    const int c0 = (grp * (D / 64) + c) * 32;
    float v[32];
    tmem_ld32(w + c0, v);
    tmem_ld_wait();
    if (krow < p.N) {   // (the load is the whole warp's)
      if (p.w_state != nullptr) store_u32(p.w_state, CASTLE_F32, ((int64_t)bh * p.N + krow) * D + c0, v);
      if (p.u_out.ptr != nullptr)
        store_u32(p.u_out.ptr, p.u_dtype, bh / p.H * p.u_out.stride_b + bh % p.H * p.u_out.stride_h + (int64_t)krow * p.u_out.stride_n + c0, v);
    }
  }
}

// S/scale = Sc/scale - silu(Su)/scale (rows i, columns k); Su comes in pieces of 16 columns, one ahead of the arithmetic
__device__ __forceinline__ void score_pass(uint32_t su, uint32_t sc, float half_scale, float (&s)[2][32]) {
  float w[2][16];
  tmem_ld16(su, w[0]);
  tmem_ld32(sc, s[0]);
  tmem_ld32(sc + 32, s[1]);
  tmem_ld_wait();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (q < 3) tmem_ld16(su + 16 * (q + 1), w[(q + 1) & 1]);
    float* sq = &s[q >> 1][(q & 1) * 16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const float2 u = make_float2(w[q & 1][j], w[q & 1][j + 1]);
      const float2 x = fma2(u, neg_sigmoid2(u, half_scale), make_float2(sq[j], sq[j + 1]));
      sq[j] = x.x; sq[j + 1] = x.y;
    }
    if (q < 3) tmem_ld_wait();
  }
}

// Causal mask of a diagonal block and the largest of the 64
__device__ __forceinline__ float masked_max(float (&s)[2][32], int row, int cbase, bool diag) {
  if (diag) {
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
      for (int j = 0; j < 32; ++j) s[c][j] = (cbase + c * 32 + j <= row) ? s[c][j] : -INFINITY;
  }
  float mx = s[0][0];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int j = 0; j < 32; ++j) mx = fmaxf(mx, s[c][j]);
  return mx;
}

// P = exp(scale * v - max) as packed pairs into tensor memory (masked entries give 0) and its sum.  An eighth of the exponentials at
// dim_head 64, where the special-function unit is the busiest (53 %), is computed on the FMA pipe: 752 -> 746 us at B=4 N=4096
// H=16; no gain at 128.
template <typename T, int D>
__device__ __forceinline__ float exp_pass(float (&s)[2][32], float sl2, float mb, uint32_t dst) {
  float2 lsum = splat(0.f);
#pragma unroll
  for (int c = 0; c < 2; ++c) {
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const float2 x = fma2(make_float2(s[c][j], s[c][j + 1]), splat(sl2), splat(-mb));
      const float2 e = D == 64 && j % 16 == 0 ? exp2_fma2(x) : make_float2(ex2_approx(x.x), ex2_approx(x.y));
      s[c][j] = e.x;
      s[c][j + 1] = e.y;
      lsum = add2(lsum, make_float2(s[c][j], s[c][j + 1]));
    }
    tmem_st_packed32<T>(dst + c * 16, s[c]);
  }
  return lsum.x + lsum.y;
}

// A group's columns of the un-normalised P @ Vc of one tile
template <typename T, int D>
__device__ __forceinline__ void store_partial(const FwdParams& p, int64_t tile, int row, int grp, const float (&o)[D / 64][32]) {
#pragma unroll
  for (int c = 0; c < D / 64; ++c) {
    uint4* dst = reinterpret_cast<uint4*>(p.part_o) + (tile * (D / 8) + (grp * (D / 64) + c) * 4) * kBlk + row;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      dst[j * kBlk] = make_uint4(Elem<T>::pack2(o[c][8 * j], o[c][8 * j + 1]), Elem<T>::pack2(o[c][8 * j + 2], o[c][8 * j + 3]),
                                 Elem<T>::pack2(o[c][8 * j + 4], o[c][8 * j + 5]), Elem<T>::pack2(o[c][8 * j + 6], o[c][8 * j + 7]));
  }
}

template <typename T, int D, bool TM>
__global__ void __launch_bounds__(kFwdThreads, 1)
castle_fwd_pipe_kernel(const FwdParams p, const __grid_constant__ CUtensorMap m_qc, const __grid_constant__ CUtensorMap m_kc,
                       const __grid_constant__ CUtensorMap m_vc, const __grid_constant__ CUtensorMap m_qu,
                       const __grid_constant__ CUtensorMap m_ku, const __grid_constant__ CUtensorMap m_vu,
                       const __grid_constant__ CUtensorMap m_quc, const __grid_constant__ CUtensorMap m_kcc,
                       const __grid_constant__ CUtensorMap m_vcc) {
  using L = FwdPipe<D>;
  constexpr int NP = D / 64;
  constexpr bool B2 = D == 64;   // two buffers of everything that is streamed
  constexpr uint32_t OPB = L::OPB;
  constexpr uint32_t C_W = 0, C_R1 = D, C_R2 = D + 128, C_R3 = D + 256;
  constexpr uint32_t C_O = B2 ? C_R3 + 64 : C_R2, C_TM = B2 ? C_R3 + 128 : C_R1;
  constexpr int FMT = Elem<T>::fmt;
  constexpr uint32_t ID_SQ = make_idesc(128, 128, FMT, false, false, false);
  constexpr uint32_t ID_D = make_idesc(128, D, FMT, false, true, false);
  constexpr float kLog2e = 1.4426950408889634f;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sQu = smem, *sKc = sQu + OPB, *sVc = sKc + OPB, *sWb = sVc + OPB, *sStream = sWb + OPB;
  // streamed tiles; n counts steps from K
  auto sKu = [&](int n) { return B2 ? sStream + 65536 + (n & 1) * OPB : sStream + OPB + (n & 1) * 32768; };
  auto sVu = [&](int n) { return B2 ? sStream + 65536 + 2 * OPB + (n & 1) * OPB : sStream + OPB + ((n + 1) & 1) * 32768; };
  auto sQc = [&](int n) { return B2 ? sStream + 65536 + 4 * OPB + (n & 1) * OPB : sStream; };
  auto sA = [&](int n) { return B2 ? sStream + (n & 1) * 32768 : sStream + OPB + (n & 1) * 32768; };
  float (*red_max)[kBlk] = reinterpret_cast<float (*)[kBlk]>(smem + L::kRed);
  float (*red_sum)[kBlk] = red_max + 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  // loads: the resident tiles and Ku of the first step; Vu[I], Qc[I] (and, with two buffers, Ku[I+1]) of a step; Ku[I+1]
  uint64_t *bar_res = bars, *bar_in = bars + 1, *bar_ku = bars + 3;
  uint64_t *bar_z = bars + 7, *bar_t = bars + 8, *bar_w = bars + 9, *bar_s = bars + 10, *bar_o = bars + 11;
  uint64_t* bar_r = bars + 12;   // Y has read R2: Su or, at dim_head 128, P @ Vc (one arrival per warp)
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + 14);
  int* abort_flag = reinterpret_cast<int*>(bars + 15);
  volatile int* abortp = abort_flag;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: uniform for the compiler, too
  const int quarter = warp & 3, grp = (warp >> 2) & 1;   // TMEM lanes 32 * quarter.., columns 64 * grp.. of a score tile
  const int row = quarter * 32 + lane, cbase = grp * 64;
  const int bh = blockIdx.x, K = blockIdx.y;
  const int b = bh / p.H, h = bh % p.H;
  const int k0 = K * kBlk;
  // Walk segments (gridDim.z parts, later ones first in the grid): the CTA of a later part first rebuilds the state it
  // would have inherited in state-only steps (Z, gate, W += A @ Vu).
  const int walk = p.nblk - K, nseg = walk >= kSplitMin ? (int)gridDim.z : 1, seg = (int)gridDim.z - 1 - (int)blockIdx.z;
  if (seg >= nseg) return;
  const int I_begin = K + walk_cut(walk, nseg, seg), I_end = K + walk_cut(walk, nseg, seg + 1);

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled tiles need 1024-byte alignment
    if (tid == 0) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < 12; ++i) mbar_init(bars + i, bars + i == bar_s ? 2 : 1);   // the scores: Su by X, Sc by Y
    mbar_init(bar_r, 8);
    mbar_fence_init();
    *abort_flag = 0;
    tma_prefetch_desc(&m_qc); tma_prefetch_desc(&m_ku); tma_prefetch_desc(&m_vu);
  }
  if (warp == 0) { tmem_alloc(tmem_base_s, 512); tmem_relinquish(); }
  overlap_wait();   // launched while the T tiles are being written
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s;
  const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
  const uint32_t aQu = smem_u32(sQu), aKc = smem_u32(sKc), aVc = smem_u32(sVc), aWb = smem_u32(sWb);
  const float half_scale = 0.5f * p.scale;

  auto load = [&](uint8_t* dst, const CUtensorMap& m, uint64_t* bar, int r0) {   // one d-wide tile
#pragma unroll
    for (int pn = 0; pn < NP; ++pn) tma_load_4d(dst + pn * kPanelBytes, &m, bar, pn * 64, r0, h, b);
  };
  // what step n reads: one barrier (two buffers: alternating)
  auto in_bar = [&](int n) { return B2 ? bar_in + (n & 1) : bar_in; };
  auto in_par = [&](int n) { return (uint32_t)(B2 ? n >> 1 : n) & 1u; };
  auto load_step = [&](int n) {
    const int I = K + n;
    const bool qc = I >= I_begin, ku = B2 && I + 1 < I_end;
    uint64_t* bar = in_bar(n);
    mbar_expect_tx(bar, OPB * (1 + qc + ku));
    if (ku) load(sKu(n + 1), m_ku, bar, (I + 1) * kBlk);
    load(sVu(n), m_vu, bar, I * kBlk);
    if (qc) load(sQc(n), m_qc, bar, I * kBlk);
  };
  // One polling lane per warp: a barrier over the group behind a single poll holds every warp up for the issuing one, and
  // 32 polling lanes take issue slots from the group that is working (735 against 820 and 751 us at B=4 N=4096 H=16).
  auto wait_warp = [&](uint64_t* bar, uint32_t parity) { if (elect_one()) mbar_wait_lazy_abort(bar, parity, abortp); __syncwarp(); tc_fence_after(); };

  if (warp < 8) {
    // ============================================================ X: lookahead stage
    if (warp == 0 && elect_one()) {
      mbar_expect_tx(bar_res, 4 * OPB);
      load(sQu, m_qu, bar_res, k0);
      load(sKu(0), m_ku, bar_res, k0);
      load_step(0);
      load(sKc, m_kc, bar_res, k0);
      load(sVc, m_vc, bar_res, k0);
      mbar_wait(bar_res, 0, abortp);
      tc_fence_after();
      gemm_kk_t<NP>(tmem + C_R1, aQu, smem_u32(sKu(0)), ID_SQ, false);
      mma_commit(bar_z);
      // Prefill hand-off: the resident tiles are the rows the decode caches hold for this key block.
      if (p.store_caches && seg == 0 && !*abortp) {
#pragma unroll
        for (int pn = 0; pn < NP; ++pn) {
          tma_store_4d(&m_quc, sQu + pn * kPanelBytes, pn * 64, k0, h, b);
          tma_store_4d(&m_kcc, sKc + pn * kPanelBytes, pn * 64, k0, h, b);
          tma_store_4d(&m_vcc, sVc + pn * kPanelBytes, pn * 64, k0, h, b);
        }
        bulk_commit();
      }
    }
    for (int I = K; I < I_end; ++I) {
      const int n = I - K;
      const bool diag = I == K, pre = I < I_begin, more = I + 1 < I_end, again = I > I_begin;
      const uint32_t ph = n & 1, ph_m = (I - I_begin) & 1;   // barriers that complete in every step; in full steps only
      const uint32_t aA = smem_u32(sA(n)), aVu = smem_u32(sVu(n)), aQc = smem_u32(sQc(n)), aKn = smem_u32(sKu(n + 1));

      uint4 tq[8];   // this thread's 64 values of the masked T, on their way during the gate
      if (TM && !pre) {
        const uint4* src = p.tm + ((int64_t)bh * p.nblk + I) * kTmTile + (cbase / 8) * kBlk + row;
#pragma unroll
        for (int q = 0; q < 8; ++q) tq[q] = __ldg(src + q * kBlk);
      }
      // ---- gate A = sigmoid(scale * Z), kept for j > k (rows k, columns j)
      wait_warp(bar_z, ph);
      PIPE_MARK(0);
      gate_pass<T>(trow + C_R1, sA(n), row, cbase, half_scale, diag);
      PIPE_MARK(1);
      if (B2) {
        // Y has the scores of the step before, so its products are done: its buffers are filled for the next one
        if (again) wait_warp(bar_r, ph_m ^ 1);
        if (more && warp == 1 && elect_one()) load_step(n + 1);
        __syncwarp();
      }
      if (!pre) state_copy<T, D>(trow + C_W, sWb, row, grp);   // before this step's update
      if (TM && !pre) {
        if (!B2) { tc_fence_before(); sync_pair(3 + quarter); tc_fence_after(); }   // the masked T goes over Z
#pragma unroll
        for (int c = 0; c < 2; ++c) tmem_st16(trow + C_TM + cbase / 2 + c * 16, reinterpret_cast<const uint32_t*>(tq + 4 * c));
        tmem_st_wait();
      }
      fence_async_smem();
      tc_fence_before();
      // what the products below read is waited for here, by another warp than the issuing one
      if (warp == 1 && elect_one()) mbar_wait_lazy_abort(in_bar(n), in_par(n), abortp);
      __syncwarp();
      sync_x();
      PIPE_MARK(2);
      if (!TM && !pre) {
        // ---- T[I,I] = Qc[I] @ Vu[I]^T over Z, masked (j <= i) into packed pairs
        if (warp == 0 && elect_one()) {
          tc_fence_after();
          gemm_kk_t<NP>(tmem + C_R1, aQc, aVu, ID_SQ, false);
          mma_commit(bar_t);
        }
        wait_warp(bar_t, ph_m);
        float v[2][32];
        tmem_ld32_lower(trow + C_R1 + cbase, row, cbase, v[0]);
        tmem_ld32_lower(trow + C_R1 + cbase + 32, row, cbase + 32, v[1]);
        if (!B2) { tc_fence_before(); sync_pair(3 + quarter); tc_fence_after(); }   // the rows' T is in registers
        tmem_st_packed32<T>(trow + C_TM + cbase / 2, v[0]);
        tmem_st_packed32<T>(trow + C_TM + cbase / 2 + 16, v[1]);
        tmem_st_wait();
        tc_fence_before();
        sync_x();
      }

      // ---- W_K += A @ Vu[I];  Su/scale = Qc[I] @ Wb^T + Tm @ A^T;  Z of the next step
      if (warp == 0 && elect_one()) {
        tc_fence_after();
        if (B2 && more && !pre) {   // R1 has been read: Z first, the next gate waits for nothing else
          gemm_kk_t<NP>(tmem + C_R1, aQu, aKn, ID_SQ, false);
          mma_commit(bar_z);
        }
        PIPE_MARK(7);
        gemm_km_t<8>(tmem + C_W, aA, aVu, ID_D, !diag);
        mma_commit(bar_w);
        PIPE_MARK(14);
        if (!pre) {
          if (!B2 && again) { mbar_wait(bar_r, ph_m ^ 1, abortp); tc_fence_after(); }
          PIPE_MARK(3);
          if (!diag) gemm_kk_t<NP>(tmem + C_R2, aQc, aWb, ID_SQ, false);
          gemm_tk_t<2>(tmem + C_R2, tmem + C_TM, aA, ID_SQ, !diag);
          mma_commit(bar_s);
          if (!again) {   // the first Sc (later ones are Y's)
            gemm_kk_t<NP>(tmem + C_R3, aQc, aKc, ID_SQ, false);
            mma_commit(bar_s);
          }
          PIPE_MARK(5);
        }
        if (more && (!B2 || pre)) {   // (state-only steps: behind the update, so that it covers the update too)
          if (!B2) { mbar_wait(bar_ku, ph, abortp); tc_fence_after(); }
          gemm_kk_t<NP>(tmem + C_R1, aQu, aKn, ID_SQ, false);
          mma_commit(bar_z);
        }
      }
      if (!B2 && more && warp == 1 && elect_one()) {
        mbar_wait(bar_w, ph, abortp);   // Vu[I] is consumed by the update: Ku[I+1] over it
        mbar_expect_tx(bar_ku, OPB);
        load(sKu(n + 1), m_ku, bar_ku, (I + 1) * kBlk);
        if (!pre) mbar_wait(bar_s, ph_m, abortp);   // the gate and Qc[I] are consumed by the scores
        load_step(n + 1);
      }
      if (!B2) __syncwarp();
    }
    // ---- W_K is now U[K] (in the CTA that walked to the last query block)
    if (I_end == p.nblk && (p.u_out.ptr != nullptr || p.w_state != nullptr)) {
      wait_warp(bar_w, (uint32_t)(I_end - 1 - K) & 1u);
      state_out<D>(p, trow + C_W, bh, K, row, grp);
    }
    if (p.store_caches && warp == 0 && elect_one()) bulk_wait0();
  } else {
    // ============================================================ Y: soft-max stage
    const float sl2 = p.scale * kLog2e;
    auto issue_sc = [&](int I) {   // Sc/scale = Qc[I] @ Kc[K]^T
      if (I < I_end && warp == 8 && elect_one()) {
        tc_fence_after();
        gemm_kk_t<NP>(tmem + C_R3, smem_u32(sQc(I - K)), aKc, ID_SQ, false);
        mma_commit(bar_s);
      }
      __syncwarp();
    };
    if (warp == 8 && elect_one()) mbar_wait(bar_res, 0, abortp);   // Kc, Vc
    __syncwarp();
    for (int I = I_begin; I < I_end; ++I) {
      const uint32_t ph_m = (I - I_begin) & 1;
      const bool diag = I == K;
      const int irow = I * kBlk + row;
      wait_warp(bar_s, ph_m);
      PIPE_MARK(8);
      float s[2][32];
      score_pass(trow + C_R2 + cbase, trow + C_R3 + cbase, half_scale, s);
      tc_fence_before();
      if (B2) {   // Su is in registers; at dim_head 128 its columns take P @ Vc first
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_r);
      }
      float mx = masked_max(s, row, cbase, diag);
      red_max[grp][row] = mx;
      PIPE_MARK(9);
      sync_pair(7 + quarter);
      tc_fence_after();
      mx = fmaxf(mx, red_max[grp ^ 1][row]);   // column 0 is never masked, so the maximum is finite
      const float mb = mx * sl2;
      red_sum[grp][row] = exp_pass<T, D>(s, sl2, mb, trow + C_R3 + cbase / 2);   // P over Sc, which everybody has read
      tmem_st_wait();
      tc_fence_before();
      sync_y();
      PIPE_MARK(10);
      // ---- O_partial = P @ Vc[K]
      if (warp == 8 && elect_one()) {
        tc_fence_after();
        gemm_tm_t<8>(tmem + C_O, tmem + C_R3, aVc, ID_D, false);
        mma_commit(bar_o);
      }
      const int64_t tile = (int64_t)bh * tri(p.nblk) + tri(I) + K;
      if (grp == 0 && irow < p.N)
        reinterpret_cast<float2*>(p.part_ml)[tile * kBlk + row] = make_float2(mx * p.scale, red_sum[0][row] + red_sum[1][row]);
      if (I + 1 < I_end && (B2 ? warp == 9 : warp == 8) && elect_one()) mbar_wait_lazy_abort(in_bar(I + 1 - K), in_par(I + 1 - K), abortp);   // Qc for the next Sc
      wait_warp(bar_o, ph_m);
      if (!B2) issue_sc(I + 1);   // over P
      PIPE_MARK(11);
      float o[NP][32];
#pragma unroll
      for (int c = 0; c < NP; ++c) tmem_ld32(trow + C_O + (grp * NP + c) * 32, o[c]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (B2) sync_y();
      else if (lane == 0) mbar_arrive(bar_r);
      PIPE_MARK(12);
      if (B2) issue_sc(I + 1);   // over P and P @ Vc, which everybody has read
      if (irow < p.N) store_partial<T, D>(p, tile, row, grp, o);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && *abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

// ---------------------------------------------------------------------------------------------
// The pipeline above at dim_head 64, for CTAs that stay on their SM and walk one key block after the other: X goes on to the next
// walk while Y is still on the last block of the one before, so that start and end of a walk, 7 to 9 us of a CTA that has but
// one (tensor memory, first tiles, the fill of the pipeline, the last block), are covered.  A step is bound by its chain, as above.
// B=16 N=1024 H=8 146 -> 124 us, B=8 N=2049 H=16 484 -> 460 us, B=64 N=512 H=8 182 -> 165 us against a CTA (or two per SM, below seven
// blocks) for each walk.
//
// Tensor memory: W | R1 (Z) | R2 (Su) | R3 (Sc, issued by Y as soon as these columns are free again, then P as packed pairs and, in
// its upper half, P @ Vc) | Tm.  Shared memory: Qu, Kc, Vc of the walk, the 16-bit copy of W, and two buffers each of Ku, Vu, Qc
// and the gate, filled a step ahead.  n counts a CTA's steps, i its walks; a barrier's parity is its count's.
struct Walk64 { int bh, K; };   // key block K of pair bh over query blocks [K, nblk)
// The steps of a CTA, walk after walk.  The walks are ordered from the longest to the shortest (key blocks upwards, each over all
// pairs) and dealt out to the CTAs back and forth, so that every CTA gets about as many steps.
struct Steps64 {
  Walk64 w;
  int I, ahead, back;   // places from this walk to the next, and from that to the one behind
  bool ok;
  __device__ __forceinline__ Steps64(const FwdParams& p) {
    const int pairs = p.B * p.H;
    I = w.K = blockIdx.x / pairs;
    w.bh = blockIdx.x % pairs;
    ok = w.K < p.nblk;
    ahead = 2 * (int)(gridDim.x - blockIdx.x) - 1;
    back = 2 * blockIdx.x + 1;
  }
  __device__ __forceinline__ void advance(const FwdParams& p) {
    if (++I < p.nblk) return;
    const int t = ahead, pairs = p.B * p.H;
    w.bh += ahead;
    ahead = back;
    back = t;
    while (w.bh >= pairs && w.K < p.nblk) { w.bh -= pairs; ++w.K; }
    ok = w.K < p.nblk;
    I = w.K;
  }
  __device__ __forceinline__ bool first() const { return I == w.K; }
};

template <typename T, bool TM>
__global__ void __launch_bounds__(kFwdThreads, 1)
castle_fwd_pipe64_kernel(const FwdParams p, const __grid_constant__ CUtensorMap m_qc, const __grid_constant__ CUtensorMap m_kc,
                         const __grid_constant__ CUtensorMap m_vc, const __grid_constant__ CUtensorMap m_qu,
                         const __grid_constant__ CUtensorMap m_ku, const __grid_constant__ CUtensorMap m_vu,
                         const __grid_constant__ CUtensorMap m_quc, const __grid_constant__ CUtensorMap m_kcc,
                         const __grid_constant__ CUtensorMap m_vcc) {
  using L = FwdPipe<64>;
  constexpr int D = 64;
  constexpr uint32_t OPB = L::OPB;
  constexpr uint32_t C_W = 0, C_R1 = D, C_R2 = D + 128, C_R3 = D + 256, C_O = C_R3 + 64, C_TM = C_R3 + 128;
  constexpr int FMT = Elem<T>::fmt;
  constexpr uint32_t ID_SQ = make_idesc(128, 128, FMT, false, false, false);
  constexpr uint32_t ID_D = make_idesc(128, D, FMT, false, true, false);
  constexpr float kLog2e = 1.4426950408889634f;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *sQu = smem, *sKc = sQu + OPB, *sVc = sKc + OPB, *sWb = sVc + OPB, *sStream = sWb + OPB;
  auto sA = [&](uint32_t n) { return sStream + (n & 1) * 32768; };
  auto sKu = [&](uint32_t n) { return sStream + 65536 + (n & 1) * OPB; };
  auto sVu = [&](uint32_t n) { return sStream + 65536 + 2 * OPB + (n & 1) * OPB; };
  auto sQc = [&](uint32_t n) { return sStream + 65536 + 4 * OPB + (n & 1) * OPB; };
  float (*red_max)[kBlk] = reinterpret_cast<float (*)[kBlk]>(smem + L::kRed);
  float (*red_sum)[kBlk] = red_max + 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBars);
  // loads: Qu, Kc, Vc of a walk; Vu and Qc of a step with Ku of the next (two, alternating); Ku of the first step
  uint64_t *bar_qu = bars, *bar_kc = bars + 1, *bar_vc = bars + 2, *bar_in = bars + 3, *bar_ku0 = bars + 5;
  uint64_t *bar_z = bars + 6, *bar_t = bars + 7, *bar_w = bars + 8, *bar_s = bars + 9, *bar_o = bars + 10;
  uint64_t* bar_r = bars + 11;   // Y has Su in registers (one arrival per warp)
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(bars + 14);
  int* abort_flag = reinterpret_cast<int*>(bars + 15);
  volatile int* abortp = abort_flag;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: uniform for the compiler, too
  const int quarter = warp & 3, grp = (warp >> 2) & 1;   // TMEM lanes 32 * quarter.., columns 64 * grp.. of a score tile
  const int row = quarter * 32 + lane, cbase = grp * 64;
  Steps64 c(p);
  if (!c.ok) return;

  if ((smem_u32(smem) & 1023u) != 0) {  // the swizzled tiles need 1024-byte alignment
    if (tid == 0) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < 11; ++i) mbar_init(bars + i, bars + i == bar_s ? 2 : 1);   // the scores: Su by X, Sc by Y
    mbar_init(bar_r, 8);
    mbar_fence_init();
    *abort_flag = 0;
    tma_prefetch_desc(&m_qc); tma_prefetch_desc(&m_ku); tma_prefetch_desc(&m_vu);
  }
  if (warp == 0) { tmem_alloc(tmem_base_s, 512); tmem_relinquish(); }
  overlap_wait();   // launched while the T tiles are being written
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s;
  const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
  const uint32_t aQu = smem_u32(sQu), aKc = smem_u32(sKc), aVc = smem_u32(sVc), aWb = smem_u32(sWb);
  const float half_scale = 0.5f * p.scale;

  auto load = [&](uint8_t* dst, const CUtensorMap& map, uint64_t* bar, int block, int bh) {
    tma_load_4d(dst, &map, bar, 0, block * kBlk, bh % p.H, bh / p.H);
  };
  // what step n reads, and Ku of the step behind it
  auto load_step = [&](uint32_t n, const Steps64& s) {
    Steps64 next = s;
    next.advance(p);
    uint64_t* bar = bar_in + (n & 1);
    mbar_expect_tx(bar, OPB * (2 + next.ok));
    if (next.ok) load(sKu(n + 1), m_ku, bar, next.I, next.w.bh);
    load(sVu(n), m_vu, bar, s.I, s.w.bh);
    load(sQc(n), m_qc, bar, s.I, s.w.bh);
  };
  // A walk's resident tile; in a prompt it is also what a decode cache holds for the key block, and is stored there as it is.  One
  // lane does all of it for a tile, so that it knows when the store has read the tile that the next load overwrites.
  auto load_resident = [&](uint8_t* dst, const CUtensorMap& map, uint64_t* bar, const Walk64& w) {
    if (p.store_caches) bulk_wait_read0();
    mbar_expect_tx(bar, OPB);
    load(dst, map, bar, w.K, w.bh);
  };
  auto resident = [&](uint8_t* tile, const CUtensorMap& cache, uint64_t* bar, uint32_t i, const Walk64& w) {
    mbar_wait_lazy_abort(bar, i & 1, abortp);
    if (p.store_caches && !*abortp) {
      tma_store_4d(&cache, tile, 0, w.K * kBlk, w.bh % p.H, w.bh / p.H);
      bulk_commit();
    }
  };
  // one polling lane per warp (see castle_fwd_pipe_kernel)
  auto wait_warp = [&](uint64_t* bar, uint32_t parity) { if (elect_one()) mbar_wait_lazy_abort(bar, parity & 1, abortp); __syncwarp(); tc_fence_after(); };

  if (warp < 8) {
    // ============================================================ X: lookahead stage
    uint32_t n = 0, i = 0;
    if (warp == 0 && elect_one()) {
      load_resident(sQu, m_qu, bar_qu, c.w);
      mbar_expect_tx(bar_ku0, OPB);
      load(sKu(0), m_ku, bar_ku0, c.w.K, c.w.bh);
      load_step(0, c);
      resident(sQu, m_quc, bar_qu, 0, c.w);
      mbar_wait(bar_ku0, 0, abortp);
      tc_fence_after();
      gemm_kk_t<1>(tmem + C_R1, aQu, smem_u32(sKu(0)), ID_SQ, false);
      mma_commit(bar_z);
    }
    Walk64 last{};
#pragma unroll 1
    while (c.ok) {
      Steps64 next = c;
      next.advance(p);
      const bool diag = c.first(), more = next.ok;
      const uint32_t aA = smem_u32(sA(n)), aVu = smem_u32(sVu(n)), aQc = smem_u32(sQc(n)), aKn = smem_u32(sKu(n + 1));

      uint4 tq[8];   // this thread's 64 values of the masked T, on their way during the gate
      if (TM) {
        const uint4* src = p.tm + ((int64_t)c.w.bh * p.nblk + c.I) * kTmTile + (cbase / 8) * kBlk + row;
#pragma unroll
        for (int q = 0; q < 8; ++q) tq[q] = __ldg(src + q * kBlk);
      }
      // ---- gate A = sigmoid(scale * Z), kept for j > k (rows k, columns j)
      wait_warp(bar_z, n);
      if (more && next.first() && warp == 0 && elect_one()) load_resident(sQu, m_qu, bar_qu, next.w);   // this Z was the last with the old one
      __syncwarp();
      gate_pass<T>(trow + C_R1, sA(n), row, cbase, half_scale, diag);
      // Y has the scores of the step before, so its products are done: its buffers are filled for the next one
      if (n > 0) wait_warp(bar_r, n - 1);
      if (more && warp == 1 && elect_one()) load_step(n + 1, next);
      __syncwarp();
      if (diag && n > 0) {   // W is U of the walk before
        if (p.u_out.ptr != nullptr || p.w_state != nullptr) state_out<D>(p, trow + C_W, last.bh, last.K, row, grp);
      } else {
        state_copy<T, D>(trow + C_W, sWb, row, grp);   // before this step's update
      }
      if (TM) {
#pragma unroll
        for (int q = 0; q < 2; ++q) tmem_st16(trow + C_TM + cbase / 2 + q * 16, reinterpret_cast<const uint32_t*>(tq + 4 * q));
        tmem_st_wait();
      }
      fence_async_smem();
      tc_fence_before();
      // what the products below read is waited for here, by another warp than the issuing one
      if (warp == 1 && elect_one()) mbar_wait_lazy_abort(bar_in + (n & 1), (n >> 1) & 1, abortp);
      __syncwarp();
      sync_x();
      if (!TM) {
        // ---- T[I,I] = Qc[I] @ Vu[I]^T over Z, masked (j <= i) into packed pairs
        if (warp == 0 && elect_one()) {
          tc_fence_after();
          gemm_kk_t<1>(tmem + C_R1, aQc, aVu, ID_SQ, false);
          mma_commit(bar_t);
        }
        wait_warp(bar_t, n);
        float v[2][32];
        tmem_ld32_lower(trow + C_R1 + cbase, row, cbase, v[0]);
        tmem_ld32_lower(trow + C_R1 + cbase + 32, row, cbase + 32, v[1]);
        tmem_st_packed32<T>(trow + C_TM + cbase / 2, v[0]);
        tmem_st_packed32<T>(trow + C_TM + cbase / 2 + 16, v[1]);
        tmem_st_wait();
        tc_fence_before();
        sync_x();
      }

      // ---- Z of the next step;  W_K += A @ Vu[I];  Su/scale = Qc[I] @ Wb^T + Tm @ A^T
      if (warp == 0 && elect_one()) {
        tc_fence_after();
        if (more) {   // R1 has been read: Z first, the next gate waits for nothing else
          if (next.first()) { resident(sQu, m_quc, bar_qu, i + 1, next.w); tc_fence_after(); }
          gemm_kk_t<1>(tmem + C_R1, aQu, aKn, ID_SQ, false);
          mma_commit(bar_z);
        }
        gemm_km_t<8>(tmem + C_W, aA, aVu, ID_D, !diag);
        mma_commit(bar_w);
        if (!diag) gemm_kk_t<1>(tmem + C_R2, aQc, aWb, ID_SQ, false);
        gemm_tk_t<2>(tmem + C_R2, tmem + C_TM, aA, ID_SQ, !diag);
        mma_commit(bar_s);
        if (n == 0) {   // the first Sc (later ones are Y's)
          mbar_wait(bar_kc, 0, abortp);
          tc_fence_after();
          gemm_kk_t<1>(tmem + C_R3, aQc, aKc, ID_SQ, false);
          mma_commit(bar_s);
        }
      }
      __syncwarp();
      if (more && next.first()) ++i;
      last = c.w;
      ++n;
      c = next;
    }
    // ---- the state of the last walk
    if (p.u_out.ptr != nullptr || p.w_state != nullptr) {
      wait_warp(bar_w, n - 1);
      state_out<D>(p, trow + C_W, last.bh, last.K, row, grp);
    }
    if (p.store_caches && warp == 0 && elect_one()) bulk_wait0();
  } else {
    // ============================================================ Y: soft-max stage
    const float sl2 = p.scale * kLog2e;
    uint32_t n = 0, i = 0;
    // Kc by warp 8, which issues its product; Vc by warp 9
    auto issue_sc = [&](uint32_t step) {   // Sc/scale = Qc[I] @ Kc[K]^T
      tc_fence_after();
      gemm_kk_t<1>(tmem + C_R3, smem_u32(sQc(step)), aKc, ID_SQ, false);
      mma_commit(bar_s);
    };
    if (warp == 8 && elect_one()) {
      load_resident(sKc, m_kc, bar_kc, c.w);
      resident(sKc, m_kcc, bar_kc, 0, c.w);
    }
    if (warp == 9 && elect_one()) load_resident(sVc, m_vc, bar_vc, c.w);
    __syncwarp();
    bool first = true;   // block of a walk
#pragma unroll 1
    while (c.ok) {
      Steps64 next = c;
      next.advance(p);
      const bool diag = c.first(), turn = next.ok && next.first();   // turn: the last block of a walk, and another one follows
      const int irow = c.I * kBlk + row;
      wait_warp(bar_s, n);
      if (turn && warp == 8 && elect_one()) load_resident(sKc, m_kc, bar_kc, next.w);   // these scores were the last with the old one
      __syncwarp();
      float s[2][32];
      score_pass(trow + C_R2 + cbase, trow + C_R3 + cbase, half_scale, s);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_r);   // Su is in registers
      float mx = masked_max(s, row, cbase, diag);
      red_max[grp][row] = mx;
      sync_pair(7 + quarter);
      tc_fence_after();
      mx = fmaxf(mx, red_max[grp ^ 1][row]);   // column 0 is never masked, so the maximum is finite
      const float mb = mx * sl2;
      red_sum[grp][row] = exp_pass<T, D>(s, sl2, mb, trow + C_R3 + cbase / 2);   // P over Sc, which everybody has read
      tmem_st_wait();
      tc_fence_before();
      if (first && warp == 9 && elect_one()) resident(sVc, m_vcc, bar_vc, i, c.w);
      __syncwarp();
      sync_y();
      // ---- O_partial = P @ Vc[K]
      if (warp == 8 && elect_one()) {
        tc_fence_after();
        gemm_tm_t<8>(tmem + C_O, tmem + C_R3, aVc, ID_D, false);
        mma_commit(bar_o);
      }
      const int64_t tile = (int64_t)c.w.bh * tri(p.nblk) + tri(c.I) + c.w.K;
      if (grp == 0 && irow < p.N)
        reinterpret_cast<float2*>(p.part_ml)[tile * kBlk + row] = make_float2(mx * p.scale, red_sum[0][row] + red_sum[1][row]);
      if (next.ok && warp == 9 && elect_one()) mbar_wait_lazy_abort(bar_in + ((n + 1) & 1), ((n + 1) >> 1) & 1, abortp);   // Qc for the next Sc
      wait_warp(bar_o, n);
      float o[1][32];
      tmem_ld32(trow + C_O + grp * 32, o[0]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (turn && warp == 9 && elect_one()) load_resident(sVc, m_vc, bar_vc, next.w);
      __syncwarp();
      sync_y();
      if (next.ok && warp == 8 && elect_one()) {   // over P and P @ Vc, which everybody has read
        if (turn) resident(sKc, m_kcc, bar_kc, i + 1, next.w);
        issue_sc(n + 1);
      }
      __syncwarp();
      if (irow < p.N) store_partial<T, D>(p, tile, row, grp, o);
      if (turn) ++i;
      first = turn;
      ++n;
      c = next;
    }
    if (p.store_caches && (warp == 8 || warp == 9) && elect_one()) bulk_wait0();
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && *abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

// The masked T tiles: one CTA of 128 threads (a row each) per query block.
template <typename T, int D>
__global__ void __launch_bounds__(128) castle_fwd_t_kernel(const FwdParams p, const __grid_constant__ CUtensorMap m_qc,
                                                           const __grid_constant__ CUtensorMap m_vu) {
  constexpr int NP = D / 64;
  constexpr uint32_t OPB = NP * kPanelBytes;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint64_t bar_in, bar_t;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int bh = blockIdx.x, I = blockIdx.y, b = bh / p.H, h = bh % p.H;
  if (tid == 0) {
    mbar_init(&bar_in, 1);
    mbar_init(&bar_t, 1);
    mbar_fence_init();
    abort_flag = 0;
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, 128); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s, trow = tmem + ((uint32_t)(warp * 32) << 16);
  if (tid == 0) {
    if (smem_u32(smem) & 1023u) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);
    mbar_expect_tx(&bar_in, 2 * OPB);
#pragma unroll
    for (int pn = 0; pn < NP; ++pn) {
      tma_load_4d(smem + pn * kPanelBytes, &m_qc, &bar_in, pn * 64, I * kBlk, h, b);
      tma_load_4d(smem + OPB + pn * kPanelBytes, &m_vu, &bar_in, pn * 64, I * kBlk, h, b);
    }
    mbar_wait(&bar_in, 0, &abort_flag);
    tc_fence_after();
    gemm_kk_t<NP>(tmem, smem_u32(smem), smem_u32(smem) + OPB, make_idesc(128, 128, Elem<T>::fmt, false, false, false), false);
    mma_commit(&bar_t);
  }
  mbar_wait(&bar_t, 0, &abort_flag);
  tc_fence_after();
  uint4* dst = p.tm + ((int64_t)bh * p.nblk + I) * kTmTile + tid;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float v[32];
    tmem_ld32_lower(trow + c * 32, tid, c * 32, v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      dst[(c * 4 + j) * kBlk] = make_uint4(Elem<T>::pack2(v[8 * j], v[8 * j + 1]), Elem<T>::pack2(v[8 * j + 2], v[8 * j + 3]),
                                           Elem<T>::pack2(v[8 * j + 4], v[8 * j + 5]), Elem<T>::pack2(v[8 * j + 6], v[8 * j + 7]));
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
  if (tid == 0 && abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

// Merge the per-key-block partials of one query block: out = sum_K e^{m_K - m} O_K / sum_K e^{m_K - m} l_K.
// One CTA per query block and 32 rows; a warp owns a chunk of eight columns of them (a lane a row), so that its loads
// are contiguous.
template <typename T, int D>
__global__ void __launch_bounds__(32 * D / 8) castle_fwd_merge_kernel(const FwdParams p) {
  const int bh = blockIdx.y, I = blockIdx.x / (kBlk / 32), r = (blockIdx.x % (kBlk / 32)) * 32 + (threadIdx.x & 31), c8 = threadIdx.x >> 5;
  const int i = I * kBlk + r;
  overlap_wait();   // launched while the partials are being written
  if (i >= p.N) return;
  const int64_t tile0 = (int64_t)bh * tri(p.nblk) + tri(I);
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + tile0 * kBlk + r;
  float m = -INFINITY;
  for (int K = 0; K <= I; ++K) m = fmaxf(m, ml[(int64_t)K * kBlk].x);
  float l = 0.f, acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = 0.f;
  const uint4* po = reinterpret_cast<const uint4*>(p.part_o) + (tile0 * (D / 8) + c8) * kBlk + r;
#pragma unroll 4
  for (int K = 0; K <= I; ++K) {
    const float2 v = ml[(int64_t)K * kBlk];
    const uint4 o = po[(int64_t)K * kBlk * (D / 8)];
    const float w = __expf(v.x - m);
    l += v.y * w;
    float2 a = Elem<T>::unpack2(o.x), b2 = Elem<T>::unpack2(o.y), c = Elem<T>::unpack2(o.z), d2 = Elem<T>::unpack2(o.w);
    acc[0] += a.x * w; acc[1] += a.y * w; acc[2] += b2.x * w; acc[3] += b2.y * w;
    acc[4] += c.x * w; acc[5] += c.y * w; acc[6] += d2.x * w; acc[7] += d2.y * w;
  }
  const float inv = 1.f / l;
  const int b = bh / p.H, h = bh % p.H;
  T* dst = reinterpret_cast<T*>(p.out.ptr) + b * p.out.stride_b + h * p.out.stride_h + (int64_t)i * p.out.stride_n + c8 * 8;
  uint4 q;
  q.x = Elem<T>::pack2(acc[0] * inv, acc[1] * inv);
  q.y = Elem<T>::pack2(acc[2] * inv, acc[3] * inv);
  q.z = Elem<T>::pack2(acc[4] * inv, acc[5] * inv);
  q.w = Elem<T>::pack2(acc[6] * inv, acc[7] * inv);
  *reinterpret_cast<uint4*>(dst) = q;
  if (c8 == 0) p.lse[(int64_t)bh * p.N + i] = m + __logf(l);
}

template <typename T, int D>
static int launch_fwd_pipe(const FwdParams& p, const CUtensorMap* maps, cudaStream_t st) {
  const FwdPlan plan = fwd_plan((int64_t)p.B * p.H, p.nblk, D);
  cudaError_t e;
  if (plan.persistent) {
    auto kernel = p.tm ? castle_fwd_pipe64_kernel<T, true> : castle_fwd_pipe64_kernel<T, false>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FwdPipe<64>::kSmem);   // per device, so on every call (cheap)
    if (e != cudaSuccess) return cuda_fail(e, "castle_fwd attribute");
    e = launch_kernel(kernel, dim3((unsigned)std::min<int64_t>(148, (int64_t)p.B * p.H * p.nblk)), kFwdThreads, FwdPipe<64>::kSmem, st, p.tm != nullptr, p,
                      maps[0], maps[1], maps[2], maps[3], maps[4], maps[5], maps[6], maps[7], maps[8]);
  } else {
    auto kernel = p.tm ? castle_fwd_pipe_kernel<T, D, true> : castle_fwd_pipe_kernel<T, D, false>;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FwdPipe<D>::kSmem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_fwd attribute");
    e = launch_kernel(kernel, dim3(p.B * p.H, p.nblk, plan.nseg), kFwdThreads, FwdPipe<D>::kSmem, st, p.tm != nullptr, p, maps[0], maps[1], maps[2],
                      maps[3], maps[4], maps[5], maps[6], maps[7], maps[8]);
  }
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_fwd launch");
}

template <typename T, int D>
static int launch_fwd(const FwdParams& p, const CUtensorMap* maps, cudaStream_t st) {
  if (p.tm) {
    constexpr size_t smem = 2 * (D / 64) * kPanelBytes;
    cudaError_t e = cudaFuncSetAttribute(castle_fwd_t_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_fwd attribute");
    castle_fwd_t_kernel<T, D><<<dim3(p.B * p.H, p.nblk), 128, smem, st>>>(p, maps[0], maps[5]);
  }
  ev_start(CASTLE_KERNEL_FWD, st);
  if (const int rc = launch_fwd_pipe<T, D>(p, maps, st)) return rc;
  ev_stop(CASTLE_KERNEL_FWD, st);
  cudaError_t e = launch_kernel(castle_fwd_merge_kernel<T, D>, dim3(p.nblk * (kBlk / 32), p.B * p.H), 32 * D / 8, 0, st, true, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_fwd launch");
}

static int check_parallel_problem(const castle_problem_t* p, const char* who) {
  if (!p) return reject("%s: null problem", who);
  if (p->batch <= 0 || p->heads <= 0 || p->seq_len <= 0) return reject("%s: empty problem", who);
  if (p->dim_head != 64 && p->dim_head != 128) return reject("%s: dim_head %d not supported (64 or 128)", who, p->dim_head);
  if (p->dtype != CASTLE_BF16 && p->dtype != CASTLE_F16) return reject("%s: dtype %d not supported (bf16, fp16)", who, p->dtype);
  if ((int64_t)p->batch * p->heads > 2147483647LL || (p->seq_len + kBlk - 1) / kBlk > 65535)
    return reject("%s: grid too large", who);
  return 0;
}

}  // namespace castle

using namespace castle;

extern "C" size_t castle_fwd_workspace_bytes(const castle_problem_t* p) {
  if (!p || p->seq_len <= 0) return 0;
  int64_t nb = (p->seq_len + kBlk - 1) / kBlk;
  int64_t tiles = (int64_t)p->batch * p->heads * tri(nb);
  size_t bytes = (size_t)(tiles * kBlk * (2 * sizeof(float) + p->dim_head * 2));  // (max, sum) fp32 + a 16-bit row
  if (nb >= kTmBlocks) bytes += (size_t)((int64_t)p->batch * p->heads * nb * kTmTile * sizeof(uint4));
  return bytes;
}

static int fwd_impl(const char* who, const castle_problem_t* p, const castle_tensor_t* qc, const castle_tensor_t* kc,
                    const castle_tensor_t* vc, const castle_tensor_t* qu, const castle_tensor_t* ku,
                    const castle_tensor_t* vu, const castle_tensor_t* out, float* lse, const castle_tensor_t* u_out,
                    int32_t u_dtype, float* w_state, const castle_tensor_t* const* caches, void* workspace,
                    size_t workspace_bytes, int32_t* status, void* stream) {
  int rc = check_parallel_problem(p, who);
  if (rc) return rc;
  const castle_tensor_t* ins[6] = {qc, kc, vc, qu, ku, vu};
  const char* names[6] = {"qc", "kc", "vc", "qu", "ku", "vu"};
  for (int i = 0; i < 6; ++i)
    if (!tensor_ok(ins[i], p->dtype, names[i], &rc)) return rc;
  if (!tensor_ok(out, p->dtype, "out", &rc)) return rc;
  if (!lse || !status) return reject("%s: lse and status must not be null", who);
  if (u_out && u_out->ptr) {
    if (u_dtype != CASTLE_BF16 && u_dtype != CASTLE_F16 && u_dtype != CASTLE_F32) return reject("%s: bad u_dtype", who);
    if (!tensor_ok(u_out, u_dtype, "u_out", &rc)) return rc;
  }
  const char* cnames[3] = {"qu_cache", "kc_cache", "vc_cache"};
  if (caches)
    for (int i = 0; i < 3; ++i)
      if (!tensor_ok(caches[i], p->dtype, cnames[i], &rc)) return rc;
  size_t need = castle_fwd_workspace_bytes(p);
  if (!workspace || workspace_bytes < need)
    return reject("%s: workspace too small (%zu < %zu bytes)", who, workspace_bytes, need);
  if (((uintptr_t)workspace) % 16) return reject("%s: workspace not 16-byte aligned", who);

  FwdParams fp;
  fp.B = p->batch; fp.H = p->heads; fp.N = p->seq_len; fp.nblk = (p->seq_len + kBlk - 1) / kBlk;
  fp.scale = p->scale;
  int64_t tiles = (int64_t)p->batch * p->heads * tri(fp.nblk);
  fp.part_ml = (float*)workspace;
  fp.part_o = fp.part_ml + tiles * kBlk * 2;  // 16-bit rows behind the fp32 (max, sum) pairs
  fp.lse = lse; fp.w_state = w_state;
  fp.u_out = (u_out && u_out->ptr) ? *u_out : castle_tensor_t{nullptr, 0, 0, 0};
  fp.u_dtype = u_dtype;
  fp.out = *out; fp.status = status;
  fp.store_caches = caches ? 1 : 0;
  fp.tm = fwd_plan((int64_t)p->batch * p->heads, fp.nblk, p->dim_head).ahead ? (uint4*)((uint8_t*)workspace + tiles * kBlk * (2 * sizeof(float) + p->dim_head * 2)) : nullptr;
#ifdef CASTLE_PHASE_TIMING
  fp.timing = (long long*)((char*)workspace + need);  // the caller leaves 2 KB beyond the partials
#endif

  CUtensorMap maps[9];
  for (int i = 0; i < 6; ++i) {
    rc = make_tmap_16bit(&maps[i], ins[i], p->dtype, p->batch, p->heads, p->seq_len, p->dim_head, kBlk, names[i]);
    if (rc) return rc;
  }
  for (int i = 0; i < 3; ++i) {
    // without caches the three maps are never used by the kernel; give them a valid encoding anyway
    const castle_tensor_t* t = caches ? caches[i] : ins[3];
    rc = make_tmap_16bit(&maps[6 + i], t, p->dtype, p->batch, p->heads, p->seq_len, p->dim_head, kBlk, cnames[i]);
    if (rc) return rc;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (p->dtype == CASTLE_BF16)
    return p->dim_head == 64 ? launch_fwd<__nv_bfloat16, 64>(fp, maps, st) : launch_fwd<__nv_bfloat16, 128>(fp, maps, st);
  return p->dim_head == 64 ? launch_fwd<__half, 64>(fp, maps, st) : launch_fwd<__half, 128>(fp, maps, st);
}

extern "C" int castle_fwd(const castle_problem_t* p, const castle_tensor_t* qc, const castle_tensor_t* kc,
                          const castle_tensor_t* vc, const castle_tensor_t* qu, const castle_tensor_t* ku,
                          const castle_tensor_t* vu, const castle_tensor_t* out, float* lse,
                          const castle_tensor_t* u_out, int32_t u_dtype, float* w_state, void* workspace,
                          size_t workspace_bytes, int32_t* status, void* stream) {
  return fwd_impl("castle_fwd", p, qc, kc, vc, qu, ku, vu, out, lse, u_out, u_dtype, w_state, nullptr, workspace,
                  workspace_bytes, status, stream);
}

extern "C" int castle_fwd_prefill(const castle_problem_t* p, const castle_tensor_t* qc, const castle_tensor_t* kc,
                                  const castle_tensor_t* vc, const castle_tensor_t* qu, const castle_tensor_t* ku,
                                  const castle_tensor_t* vu, const castle_tensor_t* out, float* lse,
                                  const castle_tensor_t* u_cache, const castle_tensor_t* qu_cache,
                                  const castle_tensor_t* kc_cache, const castle_tensor_t* vc_cache, float* w_state,
                                  void* workspace, size_t workspace_bytes, int32_t* status, void* stream) {
  if (!u_cache || !u_cache->ptr || !qu_cache || !kc_cache || !vc_cache)
    return reject("castle_fwd_prefill: the four cache tensors must not be null");
  const castle_tensor_t* caches[3] = {qu_cache, kc_cache, vc_cache};
  return fwd_impl("castle_fwd_prefill", p, qc, kc, vc, qu, ku, vu, out, lse, u_cache, p ? p->dtype : 0, w_state, caches,
                  workspace, workspace_bytes, status, stream);
}
