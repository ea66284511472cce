// CASTLE parallel backward for dim_head 128: four kernels that hand 16-bit tiles on through global memory.
//
//   kv       per key block K, query blocks I downwards: the scores (gate A, the peeled state W, T, Su, Sc), P, dS, dSu; dkc and
//            dvc in tensor memory, dqc[I] by TMA reduce.  A and dSu -> tiles.
//   reverse  per K, I downwards: G += dSu^T Qc[I]; the 16-bit copy of G before each step -> tiles.
//   la       per query block I, over K: dA = Gb Vu^T + dSu^T T, dZ (-> tiles, over A); dku[I], dvu[I] and dT summed in tensor
//            memory; at the end the masked dT's share of dvu and dqc, and all three gradients are written.
//   dqu      per K: dqu = sum over I of dZ Ku[I].
//
// Every gradient but dqc is owned by a CTA that keeps it in tensor memory.  A TMA reduce moves some 18 bytes per cycle and SM,
// so a lookahead kernel that owned a key block and reduced dku[I] and dvu[I] (128 KB a step, with dT masked and multiplied in
// every step) took 18.5 k cycles a step, 12.1 k without the reduces; reverse + la + dqu take 3.1 + 7.3 + 1.9 k, and kv, which
// no longer forms dT, 4.6 k less.  Measured on B=1 H=8 N=8190 bf16: 2365 -> 1708 us for the kernels, B=2 H=8 N=1333:
// 249 -> 182 us.  What bounds them: kv its chain of products and passes and shared memory; la and reverse the tiles, which
// come at 20 to 30 bytes per cycle and SM with one step's worth of shared memory to prefetch into; dqu HBM.
//
// Tiles of a step (I,K): A, then dZ | dSu | Gb; 32 KB each, as they lie in shared memory (128-byte swizzle).  The scratch is
// bounded (kTileScratchLimit): the (batch, head) pairs run in chunks, one launch of each kernel per chunk.
#include <algorithm>

#include "bwd_common.cuh"

namespace castle {

constexpr uint32_t kSq = 2 * kPanelB;   // a 128x128 tile: 32 KB
constexpr uint32_t kTileA = 0, kTileDsu = kSq, kTileG = 2 * kSq, kStepTiles = 3 * kSq;
constexpr int kB128Threads = 512;      // a thread: a row and 32 columns
constexpr size_t kB128Smem = 7 * kSq + 256;

// 32 values times `mul` to a row of a 16-bit tensor
template <typename T>
__device__ __forceinline__ void store_grad32(T* dst, const float* v, float mul) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 q;
    q.x = Elem<T>::pack2(v[8 * j] * mul, v[8 * j + 1] * mul);
    q.y = Elem<T>::pack2(v[8 * j + 2] * mul, v[8 * j + 3] * mul);
    q.z = Elem<T>::pack2(v[8 * j + 4] * mul, v[8 * j + 5] * mul);
    q.w = Elem<T>::pack2(v[8 * j + 6] * mul, v[8 * j + 7] * mul);
    *reinterpret_cast<uint4*>(dst + j * 8) = q;
  }
}
template <typename T>
__device__ __forceinline__ T* grad_row(const castle_tensor_t& t, int b, int h, int row, int c0) {
  return reinterpret_cast<T*>(t.ptr) + b * t.stride_b + h * t.stride_h + (int64_t)row * t.stride_n + c0;
}

__device__ __forceinline__ void load_op(uint8_t* dst, const CUtensorMap& m, uint64_t* bar, int r0, int h, int b) {
#pragma unroll
  for (int pn = 0; pn < 2; ++pn) tma_load_4d(dst + pn * kPanelB, &m, bar, pn * 64, r0, h, b);
}
__device__ __forceinline__ uint8_t* step_tiles(const BwdParams& p, int I, int K) {   // of this CTA's pair
  return p.tiles + ((int64_t)blockIdx.x * p.ntiles + (int64_t)I * (I + 1) / 2 + K) * kStepTiles;
}
// What every kernel starts with: shared memory behind the operands, barriers, tensor memory.  NBAR barriers of one arrival.
#define B128_BEGIN(OPERANDS, NBAR, COLS)                                                      \
  extern __shared__ __align__(1024) uint8_t smem[];                                            \
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + (OPERANDS));                       \
  uint32_t* const tmem_base_s = reinterpret_cast<uint32_t*>(bars + (NBAR));                    \
  volatile int* const abortp = reinterpret_cast<int*>(bars + (NBAR)) + 1;                      \
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;  \
  const int bh = p.bh0 + blockIdx.x, b = bh / p.H, h = bh % p.H;                               \
  if (tid == 0) {                                                                              \
    if (smem_u32(smem) & 1023u) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);                  \
    for (int i = 0; i < (NBAR); ++i) mbar_init(bars + i, 1);                                   \
    mbar_fence_init();                                                                         \
    *abortp = 0;                                                                               \
  }                                                                                            \
  if (warp == 0) { tmem_alloc(tmem_base_s, COLS); tmem_relinquish(); }                         \
  overlap_wait();                                                                              \
  tc_fence_before();                                                                           \
  __syncthreads();                                                                             \
  tc_fence_after();                                                                            \
  const uint32_t tmem = *tmem_base_s, trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);

#define B128_END(COLS)                                                                        \
  overlap_next();                                                                              \
  tc_fence_before();                                                                           \
  __syncthreads();                                                                             \
  if (warp == 0) tmem_dealloc(tmem, COLS);                                                     \
  if (tid == 0 && *abortp) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);

// Phase timing (debug builds only): thread 0 of CTA (0,0) stores clock64() at the phase boundaries of its first steps behind
// the workspace.
#ifdef CASTLE_PHASE_TIMING
#define B128_MARK(base, n, i) do { if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && (n) < 8) p.timing[(base) + (n) * 32 + (i)] = clock64(); } while (0)
#else
#define B128_MARK(base, n, i) do { } while (0)
#endif

// ------------------------------------------------------------------------------------------------ scores, dkc, dvc, dqc
// One chain per step, products and passes in turn:
//   Z | gate A (T under it);  W -= A Vu | T masked, Wb (T A^T under it);  Su | silu' (Sc under it) | P (dP under it);  dvc | dS, dSu;
//   dqc, dkc | staging (the next Z under it)
// Sixteen warps do the passes, one issues the products, one moves the tiles (ev_arrive).  While warp 0 issued the products and also
// worked in the passes, it waited as long as the tensor unit's queue was full and the others waited for it: step 15.2 k -> 12.9 k
// cycles, the kernel at B=1 H=8 N=8190 995 -> 884 us, B=2 H=8 N=1333 104 -> 92, B=8 H=16 N=512 141 -> 133.  What bounds it now: 10.7 k
// cycles of a step's 1.4 MB through shared memory, and the wait for Qc and Vu, whose slots the last product of a step frees.
// Every warp keeps the 96 registers of the launch, which is enough.  Shared out as 112 and 32 (castle_bwd_kernel) the issuing and the moving
// warp spilled: us of the four kernels, so / kept, 16 pairs of 1333 positions 176.2 / 174.1, 8 of 8190 1637 / 1631, 128 of 512 270.4 / 268.3,
// cut walks of 4 x 4096 and 8 x 2048 360.5 / 356.4 and 214 / 211; as 104 and 64 in between.
// Tensor memory: W | dkc | dvc | scratch.  Shared memory, seven tiles:
//   s0 Qu, then Wb | s1 Ku, A, dS | s2 Vu, T, P | s3 Qc | s4 Kc | s5 Vc, staging | s6 dO, dSu, staging
// with the roles of s1 and s2 exchanged in every other step: P dies first, so that the next Ku lands over it and the next Z runs
// while dqc is staged.
// TMA works its queue off in order, and a reduce moves some 18 bytes a cycle: a load queued behind the 64 KB of dqc waits
// 3.6 k cycles.  So the loads that the next step starts with (Qu, Ku, Vu, Qc) are issued before the reduces, and what is
// staged over are the tiles that it needs last: dO, and Vc, which is loaded again for that.
// Few pairs: the grid is little more than a wave, whose length is the walk of key block 0, while the mean walk is about half as
// long.  So long walks are cut in two parts of about equal cost, a CTA each (kv_split).  The second part first peels the state down
// to where it begins, in steps of Z, gate and W alone, some 0.3 of a step each: with a cut after x of n steps both cost x = n / 1.7.
// Each part leaves its fp32 sums of dkc and dvc, as they lie in shared memory, and a kernel of its own adds the two.
__host__ __device__ inline int kv_cut(int walk) { return (int)((float)walk * (1.f / 1.7f) + 0.5f); }
constexpr uint32_t kPartSum = 4 * kPanelB, kPart = 2 * kPartSum;   // 128 x 128 floats in four panels of 32 columns; dkc and dvc
__device__ __forceinline__ uint8_t* kv_part(const BwdParams& p, int bh, int K, int part) {
  return reinterpret_cast<uint8_t*>(p.acc_dvu) + ((int64_t)(bh * p.kv_split + K) * 2 + part) * kPart;
}

enum KvBar { kKvRes, kKvZin /* Qu, Ku */, kKvIn /* Qc, Vu */, kKvDo /* Vc, dO */, kKvZ, kKvT, kKvW, kKvSu, kKvSc, kKvDp, kKvDv, kKvX0, kKvX, kKvK,
             kKvCopied /* dSu */, kKvEnd /* no product is in flight */, kKvBars };
static_assert(7 * kSq + kKvBars * 8 + 12 <= kB128Smem, "barriers, the address of tensor memory, the abort flag and a zero");
// The events of a step with scores that the issuing warp takes (ev_arrive), in their order; they take turns on five named barriers.
enum KvEvent { kKvReadZ, kKvGate, kKvMaskedT, kKvCopyW, kKvReadSu, kKvReadSc, kKvP, kKvDs, kKvReadX, kKvEvents };
__device__ constexpr int kv_event(int k) { return 1 + k % 5; }
__device__ constexpr int kv_gate_alone(int n) { return 6 + (n & 1); }   // that of a step without scores
__device__ constexpr int kv_staged(int m) { return 8 + (m & 1); }       // that which the moving warp takes
constexpr int kKvGroups = 10;                                           // the chunk groups among themselves: 10 to 13

template <typename T, bool CUT>
__global__ void __launch_bounds__(kSplitThreads, 1)
castle_bwd128_kv_kernel(const BwdParams p, const __grid_constant__ CUtensorMap m_qc, const __grid_constant__ CUtensorMap m_kc,
                        const __grid_constant__ CUtensorMap m_vc, const __grid_constant__ CUtensorMap m_qu,
                        const __grid_constant__ CUtensorMap m_ku, const __grid_constant__ CUtensorMap m_vu,
                        const __grid_constant__ CUtensorMap m_do, const __grid_constant__ CUtensorMap m_acc_dqc) {
  constexpr int FMT = Elem<T>::fmt;
  constexpr uint32_t C_W = 0, C_DKC = 128, C_DVC = 256, C_S = 384;
  constexpr uint32_t ID_KK = make_idesc(128, 128, FMT, false, false, false), ID_KM = make_idesc(128, 128, FMT, false, true, false),
                     ID_KM_NEG = make_idesc(128, 128, FMT, false, true, true), ID_MM = make_idesc(128, 128, FMT, true, true, false);
  constexpr float kLog2e = 1.4426950408889634f;
  // CUT: two CTAs per key block in the grid; of a key block that is not cut the second has nothing to do
  const int K = CUT ? blockIdx.y >> 1 : blockIdx.y, part = CUT ? blockIdx.y & 1 : 0, k0 = K * kBlkB, walk = p.nblk - K;
  const bool cut = CUT && K < p.kv_split;
  if (part && !cut) return;
  const int begin = part ? kv_cut(walk) : 0, end = cut && !part ? kv_cut(walk) : walk;   // steps with scores; state alone before them
  // the slot of Ku, A, dS and that of Vu, T, P change places from step to step
  auto slot_k = [](int n) { return (n & 1 ? 2u : 1u) * kSq; };
  auto slot_v = [](int n) { return (n & 1 ? 1u : 2u) * kSq; };
  constexpr uint32_t S0 = 0, S3 = 3 * kSq, S4 = 4 * kSq, S5 = 5 * kSq, S6 = 6 * kSq;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + 7 * kSq);
  uint32_t* const tmem_base_s = reinterpret_cast<uint32_t*>(bars + kKvBars);
  volatile int* const abortp = reinterpret_cast<int*>(bars + kKvBars) + 1;
  float* const zero_s = reinterpret_cast<float*>(bars + kKvBars + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int bh = p.bh0 + blockIdx.x, b = bh / p.H, h = bh % p.H;
  // What B128_BEGIN does, from the moving warp, which can then ask for the first tiles ahead of the barrier below, as the passes do for
  // the state; nothing in flight writes what they read (only tiles, sums and gradients are being written by the kernels before this one).
  if (warp == kSplitWorkers / 32 + 1 && elect_one()) {
    if (smem_u32(smem) & 1023u) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);
    for (int i = 0; i < kKvBars; ++i) mbar_init(bars + i, i == kKvDp ? 2 : 1);   // dP: the product, and the copy of the gate that dS goes over
    mbar_fence_init();
    *abortp = 0;
    *zero_s = 0.f;
    const int il = (p.nblk - 1) * kBlkB;
    mbar_expect_tx(bars + kKvZin, 2 * kSq);
    load_op(smem + S0, m_qu, bars + kKvZin, k0, h, b);
    load_op(smem + slot_k(0), m_ku, bars + kKvZin, il, h, b);
    mbar_expect_tx(bars + kKvIn, begin == 0 ? 2 * kSq : kSq);
    if (begin == 0) load_op(smem + S3, m_qc, bars + kKvIn, il, h, b);
    load_op(smem + slot_v(0), m_vu, bars + kKvIn, il, h, b);
    mbar_expect_tx(bars + kKvRes, kSq);
    load_op(smem + S4, m_kc, bars + kKvRes, k0, h, b);
    mbar_expect_tx(bars + kKvDo, 2 * kSq);
    load_op(smem + S5, m_vc, bars + kKvDo, k0, h, b);
    load_op(smem + S6, m_do, bars + kKvDo, il - begin * kBlkB, h, b);
  }
  __syncwarp();
  float w0[32];   // of the forward's final state
  if (warp < kSplitWorkers / 32) {
    const int krow = k0 + (warp & 3) * 32 + lane;
    const float* src = p.w_state + ((int64_t)bh * p.N + krow) * 128 + (warp >> 2) * 32;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      const float4 q = (krow < p.N) ? *reinterpret_cast<const float4*>(src + j) : make_float4(0.f, 0.f, 0.f, 0.f);
      w0[j] = q.x; w0[j + 1] = q.y; w0[j + 2] = q.z; w0[j + 3] = q.w;
    }
  }
  if (warp == 0) { tmem_alloc(tmem_base_s, 512); tmem_relinquish(); }
  overlap_wait();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_base_s, trow = tmem + ((uint32_t)((warp & 3) * 32) << 16);

  if (warp >= kSplitWorkers / 32) {
    if (warp == kSplitWorkers / 32) {
      // ---- the products, in the order that the passes need them
      auto at = [&](uint32_t off) {   // made where it is used: kept in registers over the step the addresses would be spilled
        uint32_t base = smem_u32(smem);
        asm volatile("" : "+r"(base));
        return base + off;
      };
      auto next_on = [&](int id) {
        __syncwarp();
        ev_wait(id, kSplitWorkers);
        tc_fence_after();
      };
      auto next = [&](int k) { next_on(kv_event(k)); };
      auto issue_z = [&](int n) {     // Z = Qu[K] Ku[I]^T
        mbar_wait(bars + kKvZin, n & 1, abortp);
        tc_fence_after();
        gemm_kk_t<2>(tmem + C_S, at(S0), at(slot_k(n)), ID_KK, false);
        mma_commit(bars + kKvZ);
      };
      if (elect_one()) issue_z(0);
#pragma unroll 1
      for (int n = 0; n < end; ++n) {
        const int m = n - begin;
        const uint32_t ph = n & 1, ph_m = m & 1, sK = slot_k(n), sV = slot_v(n);
        const bool diag = n == walk - 1, more = n + 1 < end;
        if (CUT && m < 0) {
          next_on(kv_gate_alone(n));
          if (elect_one()) {
            mbar_wait(bars + kKvIn, ph, abortp);
            tc_fence_after();
            gemm_km_t<8>(tmem + C_W, at(sK), at(sV), ID_KM_NEG, true);   // W -= A Vu alone
            mma_commit(bars + kKvW);
            issue_z(n + 1);
          }
          continue;
        }
        next(kKvReadZ);
        if (elect_one()) {
          mbar_wait(bars + kKvIn, ph, abortp);
          tc_fence_after();
          gemm_kk_t<2>(tmem + C_S, at(S3), at(sV), ID_KK, false);        // T = Qc Vu^T, while the gate is formed
          mma_commit(bars + kKvT);
        }
        next(kKvGate);
        if (elect_one()) {
          if (!diag) gemm_km_t<8>(tmem + C_W, at(sK), at(sV), ID_KM_NEG, true);   // W -= A Vu; at the diagonal block nothing reads it
          mma_commit(bars + kKvW);
        }
        next(kKvMaskedT);
        if (elect_one()) gemm_kk_t<2>(tmem + C_S, at(sV), at(sK), ID_KK, false);  // Su/scale = T A^T + Qc Wb^T, while W is copied
        next(kKvCopyW);
        if (elect_one()) {
          if (!diag) gemm_kk_t<2>(tmem + C_S, at(S3), at(S0), ID_KK, true);
          mma_commit(bars + kKvSu);
        }
        next(kKvReadSu);
        if (elect_one()) {
          if (m == 0) mbar_wait(bars + kKvRes, 0, abortp);
          tc_fence_after();
          gemm_kk_t<2>(tmem + C_S, at(S3), at(S4), ID_KK, false);        // Sc/scale = Qc Kc^T, while silu' is formed
          mma_commit(bars + kKvSc);
        }
        next(kKvReadSc);
        if (elect_one()) {
          mbar_wait(bars + kKvDo, ph_m, abortp);
          tc_fence_after();
          gemm_kk_t<2>(tmem + C_S, at(S6), at(S5), ID_KK, false);        // dP = dO Vc^T, while P is formed
          mma_commit(bars + kKvDp);
        }
        next(kKvP);
        if (elect_one()) {
          gemm_mm_t<8>(tmem + C_DVC, at(sV), at(S6), ID_MM, m > 0);      // dvc += P^T dO, while dS is formed
          mma_commit(bars + kKvDv);
        }
        next(kKvDs);       // and dSu
        if (elect_one()) {
          if (!diag) gemm_km_t<8>(tmem + C_S, at(S6), at(S0), ID_KM, false);   // dqc = dSu Wb + dS Kc
          mma_commit(bars + kKvX0);
          gemm_km_t<8>(tmem + C_S, at(sK), at(S4), ID_KM, !diag);
          mma_commit(bars + kKvX);
          gemm_mm_t<8>(tmem + C_DKC, at(sK), at(S3), ID_MM, m > 0);      // dkc += dS^T Qc
          mma_commit(bars + kKvK);
        }
        next(kKvReadX);    // dqc
        if (more && elect_one()) issue_z(n + 1);
      }
      __syncwarp();
      if (elect_one()) {
        mma_commit(bars + kKvEnd);
        mbar_drain(bars + kKvEnd, 0);
      }
      __syncwarp();
    } else if (warp == kSplitWorkers / 32 + 1) {
      // ---- the tiles
      auto failed = [&](int bar, uint32_t parity) { return mbar_wait_failed(bars + bar, parity, abortp); };
      int n = 0, done = 0;   // a wait that did not end well ended the walk, after so many of its step
#pragma unroll 1
      for (; n < end; ++n, done = 0) {
        const int m = n - begin, i0 = (p.nblk - 1 - n) * kBlkB, in0 = i0 - kBlkB;
        const uint32_t ph = n & 1, ph_m = m & 1;
        const bool more = n + 1 < end;
        uint8_t *const tile = step_tiles(p, p.nblk - 1 - n, K), *const sK = smem + slot_k(n), *const sV = smem + slot_v(n);
        if (failed(kKvW, ph)) break;   // the gate is there
        if (CUT && m < 0) {         // the next step's tiles land over both, which are consumed, Qu stays
          if (elect_one()) {
            mbar_expect_tx(bars + kKvZin, kSq);
            load_op(sV, m_ku, bars + kKvZin, in0, h, b);
            mbar_expect_tx(bars + kKvIn, m == -1 ? 2 * kSq : kSq);
            if (m == -1) load_op(smem + S3, m_qc, bars + kKvIn, in0, h, b);
            load_op(sK, m_vu, bars + kKvIn, in0, h, b);
          }
          __syncwarp();
          continue;
        }
        if (elect_one()) {
          bulk_s2g(tile + kTileA, sK, kSq);
          bulk_commit();
          if (m > 0) {
            bulk_wait_read1();                      // the reduces of the step before have read their panels
            mbar_expect_tx(bars + kKvDo, 2 * kSq);
            load_op(smem + S5, m_vc, bars + kKvDo, k0, h, b);
            load_op(smem + S6, m_do, bars + kKvDo, i0, h, b);
          }
          bulk_wait_read0();
          mbar_arrive(bars + kKvDp);                // dS may go over the gate
        }
        __syncwarp();
        done = 1;
        if (failed(kKvDv, ph_m)) break;
        if (more && elect_one()) {
          mbar_expect_tx(bars + kKvZin, 2 * kSq);
          mbar_expect_tx(bars + kKvIn, 2 * kSq);
          load_op(sV, m_ku, bars + kKvZin, in0, h, b);   // over P
        }
        __syncwarp();
        done = 2;
        if (failed(kKvX0, ph_m)) break;
        if (elect_one()) {
          if (more) load_op(smem + S0, m_qu, bars + kKvZin, k0, h, b);
          bulk_s2g(tile + kTileDsu, smem + S6, kSq);       // behind what the next product waits for
          bulk_commit();
        }
        __syncwarp();
        if (failed(kKvK, ph_m)) break;
        if (elect_one()) {
          if (more) {                               // before the reduces, which loads would queue behind
            load_op(smem + S3, m_qc, bars + kKvIn, in0, h, b);
            load_op(sK, m_vu, bars + kKvIn, in0, h, b);
          }
          bulk_wait_read0();
          mbar_arrive(bars + kKvCopied);            // dqc may be staged over dSu
        }
        __syncwarp();
        ev_wait(kv_staged(m), kSplitWorkers);
        if (elect_one()) {
#pragma unroll
          for (int c = 0; c < 4; ++c) tma_reduce_add_3d(&m_acc_dqc, smem + S5 + c * kPanelB, c * 32, i0, bh);
          bulk_commit();
        }
        __syncwarp();
      }
      if (elect_one()) {
        if (*abortp) {   // tiles that were asked for and that nobody may have waited for must not land after the CTA has left
          const int last = n < end ? n : end - 1, next = done == 2 && last + 1 < end ? last + 1 : last;
          const int last_do = last - begin - (n < end && done == 0 ? 1 : 0);
          mbar_drain(bars + kKvRes, 0);
          mbar_drain(bars + kKvZin, next & 1);   // (these two run into their limit where they were asked for in part)
          mbar_drain(bars + kKvIn, next & 1);
          mbar_drain(bars + kKvDo, last_do > 0 ? last_do & 1 : 0);
        }
        bulk_wait_read0();   // tiles and sums are complete when the kernel is
      }
      __syncwarp();
      for (; n < end; ++n)   // nothing is asked for any more, for a barrier's last phase may still be open
        if (n >= begin) ev_wait(kv_staged(n - begin), kSplitWorkers);
    }
  } else {
    const int row = (warp & 3) * 32 + lane, cc = warp >> 2, c0 = cc * 32, krow = k0 + row;
    const float sl2 = p.scale * kLog2e, half_scale = 0.5f * p.scale;
    bool failed;
    auto wait = [&](int bar, uint32_t ph) {
      failed = mbar_wait_failed(bars + bar, ph, abortp);   // the flag on every 64th poll: B=2 H=8 N=1333 95.2 -> 92.3 us (one polling lane a warp: 100.7)
      tc_fence_after();
    };
    // a wait that did not end well ends the walk; `arrived`: the events of this step that the warp has arrived on before
#define KV_CHECK(ARRIVED) if (failed) { arrived = ARRIVED; goto stopped; }
    auto read = [&](int k) { return ev_arrive_read(kv_event(k), kSplitWorkers, zero_s); };
    auto stored_on = [&](int id) {
      fence_async_smem();
      tc_fence_before();
      ev_arrive(id, kSplitWorkers);
    };
    auto stored = [&](int k) { stored_on(kv_event(k)); };
    int n = 0;
    uint32_t arrived = 0;
    tmem_st32(trow + C_W + c0, w0);
    tmem_st_wait();
#pragma unroll 1
    for (; n < end; ++n) {
      const int m = n - begin;                    // of the steps with scores
      const uint32_t ph = n & 1, ph_m = m & 1;    // barriers that complete in every step; in steps with scores
      const int I = p.nblk - 1 - n, irow = I * kBlkB + row;
      const bool diag = I == K, rvalid = irow < p.N;
      uint8_t *const sK = smem + slot_k(n), *const sV = smem + slot_v(n);
      B128_MARK(0, n, 0);
      wait(kKvZ, ph);
      B128_MARK(0, n, 1);
      {
        float v[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        KV_CHECK(kKvReadZ)
        float hs = half_scale;
        if (!CUT || m >= 0) hs += read(kKvReadZ);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 a = sigmoid2(make_float2(v[j], v[j + 1]), hs);
          v[j] = a.x; v[j + 1] = a.y;
        }
        if (diag) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = (c0 + j > row) ? v[j] : 0.f;
        }
        store_row32<T>(sK, kPanelB, row, c0, v);
      }
      if (CUT && m < 0) {
        stored_on(kv_gate_alone(n));
        continue;
      }
      stored(kKvGate);
      B128_MARK(0, n, 2);
      wait(kKvT, ph_m);
      {  // T over Vu, which the state has then read
        float v[32];
        tmem_ld32_lower(trow + C_S + c0, row, c0, v);
        KV_CHECK(kKvMaskedT)
        wait(kKvW, ph);
        B128_MARK(0, n, 3);
        store_row32<T>(sV, kPanelB, row, c0, v);
        KV_CHECK(kKvMaskedT)
      }
      stored(kKvMaskedT);
      if (!diag) {   // Wb over Qu
        float v[32];
        tmem_ld32(trow + C_W + c0, v);
        tmem_ld_wait();
        store_row32<T>(smem + S0, kPanelB, row, c0, v);
      }
      stored(kKvCopyW);
      B128_MARK(0, n, 4);
      // loaded here, not at the top of the step, where the wait for Z is short
      const float lse_i = rvalid ? p.lse[(int64_t)bh * p.N + irow] : 0.f, delta_i = rvalid ? p.delta[(int64_t)bh * p.N + irow] : 0.f;
      wait(kKvSu, ph_m);
      B128_MARK(0, n, 5);
      uint32_t dpk[16], ppk[16];
      {
        float v[32], w[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        KV_CHECK(kKvReadSu)
        const float hs = half_scale + read(kKvReadSu);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 u = make_float2(v[j], v[j + 1]);
          const float2 g = sigmoid2(u, hs);
          // silu'(su) = g + silu(su) (1 - g)
          const float2 q = mul2(mul2(u, g), splat(-1.f));   // -silu(su) / scale
          v[j] = q.x; v[j + 1] = q.y;
          const float2 d = fma2(mul2(q, splat(-p.scale)), fma2(g, splat(-1.f), splat(1.f)), g);
          dpk[j / 2] = Elem<T>::pack2(d.x, d.y);
        }
        B128_MARK(0, n, 6);
        wait(kKvSc, ph_m);
        B128_MARK(0, n, 7);
        tmem_ld32(trow + C_S + c0, w);
        tmem_ld_wait();
        KV_CHECK(kKvReadSc)
        const float s2 = sl2 + read(kKvReadSc);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 x = fma2(add2(make_float2(w[j], w[j + 1]), make_float2(v[j], v[j + 1])), splat(s2), splat(-lse_i * kLog2e));
          v[j] = ex2_approx(x.x); v[j + 1] = ex2_approx(x.y);
        }
        if (diag) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = (c0 + j <= row) ? v[j] : 0.f;
        }
        if (!rvalid) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 32; j += 2) ppk[j / 2] = Elem<T>::pack2(v[j], v[j + 1]);
        store_row32<T>(sV, kPanelB, row, c0, v);   // P, over T
      }
      stored(kKvP);
      B128_MARK(0, n, 8);
      wait(kKvDp, ph_m);
      B128_MARK(0, n, 9);
      {
        float v[32], w[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        KV_CHECK(kKvDs)
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 ds = mul2(Elem<T>::unpack2(ppk[j / 2]), add2(make_float2(v[j], v[j + 1]), splat(-delta_i)));
          const float2 du = mul2(ds, Elem<T>::unpack2(dpk[j / 2]));
          v[j] = ds.x; v[j + 1] = ds.y;
          w[j] = -du.x; w[j + 1] = -du.y;
        }
        store_row32<T>(sK, kPanelB, row, c0, v);   // dS
        wait(kKvDv, ph_m);
        store_row32<T>(smem + S6, kPanelB, row, c0, w);   // dSu, over dO
        KV_CHECK(kKvDs)
      }
      stored(kKvDs);
      B128_MARK(0, n, 10);
      wait(kKvX, ph_m);
      B128_MARK(0, n, 11);
      // ---- dqc staged over Vc and dSu
      float v[32];
      tmem_ld32(trow + C_S + c0, v);
      tmem_ld_wait();
      KV_CHECK(kKvReadX)
      read(kKvReadX);
      if (cc >= 2) {
        wait(kKvCopied, ph_m);
        KV_CHECK(kKvEvents)
      }
      store_row32_f32(smem + S5 + cc * kPanelB, row, v);
      fence_async_smem();
      ev_arrive(kv_staged(m), kSplitWorkers);
      B128_MARK(0, n, 12);
    }
#undef KV_CHECK
  stopped:
    for (; n < end; ++n, arrived = 0) {   // what is left of the events
      if (CUT && n < begin) {
        ev_wait(kv_gate_alone(n), kSplitWorkers);
        continue;
      }
#pragma unroll 1
      for (; arrived < kKvEvents; ++arrived) ev_wait(kv_event((int)arrived), kSplitWorkers);
      ev_wait(kv_staged(n - begin), kSplitWorkers);
    }
    wait(kKvK, (uint32_t)(end - begin - 1) & 1u);
    float v[32], w[32];
    tmem_ld32(trow + C_DKC + c0, v);
    tmem_ld32(trow + C_DVC + c0, w);
    tmem_ld_wait();
    if (cut) {   // over Qu to Qc, which every product has read
      uint8_t *pk = smem + S0 + cc * kPanelB, *pv = smem + 2 * kSq + cc * kPanelB;
      store_row32_f32(pk, row, v);
      store_row32_f32(pv, row, w);
      fence_async_smem();
      group_sync(kKvGroups + cc);
      if ((warp & 3) == 1 && elect_one()) {
        uint8_t* dst = kv_part(p, bh, K, part) + cc * kPanelB;
        bulk_s2g(dst, pk, kPanelB);
        bulk_s2g(dst + kPartSum, pv, kPanelB);
        bulk_commit();
        bulk_wait_read0();
      }
      __syncwarp();
    } else if (krow < p.N) {
      store_grad32<T>(grad_row<T>(p.dkc, b, h, krow, c0), v, p.scale);
      store_grad32<T>(grad_row<T>(p.dvc, b, h, krow, c0), w, 1.f);
    }
  }
  B128_END(512)
}

// dkc and dvc of the key blocks that were walked in two parts: a block of 256 threads sums 16 rows of both.
template <typename T>
__global__ void __launch_bounds__(256) castle_bwd128_parts_kernel(const BwdParams p) {
  const int bh = p.bh0 + blockIdx.x, K = blockIdx.y, b = bh / p.H, h = bh % p.H;
  const int row = blockIdx.z * 16 + (threadIdx.x >> 4), c8 = threadIdx.x & 15, krow = K * kBlkB + row;
  overlap_wait();
  if (krow >= p.N) return;
  const uint32_t at = (c8 >> 2) * kPanelB, chunk = (c8 & 3) * 2;   // eight columns: two 16-byte chunks of a panel's row
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t off = t * kPartSum + at + swz_off(row, chunk + q);
      const float4 x = *reinterpret_cast<const float4*>(kv_part(p, bh, K, 0) + off), y = *reinterpret_cast<const float4*>(kv_part(p, bh, K, 1) + off);
      v[4 * q] = x.x + y.x; v[4 * q + 1] = x.y + y.y; v[4 * q + 2] = x.z + y.z; v[4 * q + 3] = x.w + y.w;
    }
    const float mul = t == 0 ? p.scale : 1.f;
    uint4 o;
    o.x = Elem<T>::pack2(v[0] * mul, v[1] * mul); o.y = Elem<T>::pack2(v[2] * mul, v[3] * mul);
    o.z = Elem<T>::pack2(v[4] * mul, v[5] * mul); o.w = Elem<T>::pack2(v[6] * mul, v[7] * mul);
    *reinterpret_cast<uint4*>(grad_row<T>(t == 0 ? p.dkc : p.dvc, b, h, krow, c8 * 8)) = o;
  }
}

// ------------------------------------------------------------------------------------------------ reverse state
// Step m adds query block I = nblk-1-m to G and hands the copy to step (I-1, K).  Two buffers of everything.
template <typename T>
__global__ void __launch_bounds__(kB128Threads, 1)
castle_bwd128_reverse_kernel(const BwdParams p, const __grid_constant__ CUtensorMap m_qc) {
  constexpr uint32_t ID_MM = make_idesc(128, 128, Elem<T>::fmt, true, true, false);
  const int K = blockIdx.y, steps = p.nblk - 1 - K;
  B128_BEGIN(6 * kSq, 4, 128)
  uint64_t *bar_in = bars, *bar_g = bars + 2;   // two each
  const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
  const bool loader = warp == 4, storer = warp == 8;
  auto load = [&](int m) {
    uint8_t* dst = smem + (m & 1) * 2 * kSq;
    const int I = p.nblk - 1 - m;
    mbar_expect_tx(bar_in + (m & 1), 2 * kSq);
    bulk_g2s(dst, step_tiles(p, I, K) + kTileDsu, kSq, bar_in + (m & 1));
    load_op(dst + kSq, m_qc, bar_in + (m & 1), I * kBlkB, h, b);
  };
  auto product = [&](int m) {
    const uint32_t a = smem_u32(smem + (m & 1) * 2 * kSq);
    mbar_wait(bar_in + (m & 1), (uint32_t)(m >> 1) & 1u, abortp);
    tc_fence_after();
    gemm_mm_t<8>(tmem, a, a + kSq, ID_MM, m > 0);
    mma_commit(bar_g + (m & 1));
  };
  if (loader && elect_one())
    for (int m = 0; m < steps && m < 2; ++m) load(m);
  if (warp == 0 && steps > 0 && elect_one()) product(0);
  __syncwarp();
  for (int m = 0; m < steps; ++m) {
    uint8_t* gb = smem + (4 + (m & 1)) * kSq;
    mbar_wait(bar_g + (m & 1), (uint32_t)(m >> 1) & 1u, abortp);
    tc_fence_after();
    float v[32];
    tmem_ld32(trow + c0, v);
    tmem_ld_wait();
    if (storer && elect_one()) bulk_wait_read1();   // of the copy made two steps ago
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0 && m + 1 < steps && elect_one()) product(m + 1);
    if (loader && m + 2 < steps && elect_one()) load(m + 2);
    __syncwarp();
    store_row32<T>(gb, kPanelB, row, c0, v);
    fence_async_smem();
    __syncthreads();
    if (storer && elect_one()) {
      bulk_s2g(step_tiles(p, p.nblk - 2 - m, K) + kTileG, gb, kSq);
      bulk_commit();
    }
    __syncwarp();
  }
  if (storer && elect_one()) bulk_wait_read0();
  __syncwarp();
  B128_END(128)
}

// ------------------------------------------------------------------------------------------------ dku, dvu, dT, dqc
// 16 warps for the passes and one that moves tiles: a tile's slot is filled again as soon as its last reader is done, so the
// products are ordered by what they free (Gb first): 1737 -> 1708 us of backward at N=8190 H=8 against loads issued by one of
// the 16 warps after its pass.
__device__ __forceinline__ void sync_passes() {
  fence_async_smem();
  tc_fence_before();
  asm volatile("bar.sync 1, 512;" ::: "memory");
}
template <typename T>
__global__ void __launch_bounds__(kB128Threads + 32, 1)
castle_bwd128_la_kernel(const BwdParams p, const __grid_constant__ CUtensorMap m_qc, const __grid_constant__ CUtensorMap m_qu,
                       const __grid_constant__ CUtensorMap m_vu) {
  constexpr int FMT = Elem<T>::fmt;
  constexpr uint32_t C_DKU = 0, C_DVU = 128, C_DT = 256, C_DA = 384;
  constexpr uint32_t ID_KK = make_idesc(128, 128, FMT, false, false, false), ID_KM = make_idesc(128, 128, FMT, false, true, false),
                     ID_MM = make_idesc(128, 128, FMT, true, true, false);
  const int I = p.nblk - 1 - blockIdx.y, i0 = I * kBlkB;   // the longest walks first
  const bool last = I == p.nblk - 1;                       // no G there yet
  B128_BEGIN(7 * kSq, 10, 512)
  uint8_t *sVu = smem, *sT = smem + kSq, *sA = smem + 2 * kSq, *sS = smem + 3 * kSq, *sG = smem + 4 * kSq, *sQu = smem + 5 * kSq,
          *sZ = smem + 6 * kSq;
  uint64_t *bar_res = bars, *bar_in = bars + 1, *bar_qu = bars + 2, *bar_da = bars + 3, *bar_v = bars + 4, *bar_k = bars + 5, *bar_t = bars + 6,
           *bar_g = bars + 7, *bar_p = bars + 8, *bar_zf = bars + 9;
  const int row = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
  if (warp == 16) {
    if (elect_one()) {
      auto load_qu = [&](int K) {
        mbar_expect_tx(bar_qu, kSq);
        load_op(sQu, m_qu, bar_qu, K * kBlkB, h, b);
      };
      mbar_expect_tx(bar_res, 2 * kSq);
      load_op(sVu, m_vu, bar_res, i0, h, b);
      load_op(sZ, m_qc, bar_res, i0, h, b);
      const uint32_t bytes = last ? 2 * kSq : 3 * kSq;
      mbar_expect_tx(bar_in, bytes);
      if (!last) bulk_g2s(sG, step_tiles(p, I, 0) + kTileG, kSq, bar_in);
      bulk_g2s(sS, step_tiles(p, I, 0) + kTileDsu, kSq, bar_in);
      bulk_g2s(sA, step_tiles(p, I, 0) + kTileA, kSq, bar_in);
      load_qu(0);
      for (int K = 0; K <= I; ++K) {
        const uint32_t ph = K & 1;
        const bool more = K < I;
        const uint8_t* next = step_tiles(p, I, K + 1);
        if (more) {
          mbar_wait_lazy_abort(last ? bar_v : bar_g, ph, abortp);
          mbar_expect_tx(bar_in, bytes);
          if (!last) {
            bulk_g2s(sG, next + kTileG, kSq, bar_in);
            mbar_wait_lazy_abort(bar_v, ph, abortp);
          }
          bulk_g2s(sS, next + kTileDsu, kSq, bar_in);
        }
        mbar_wait_lazy_abort(bar_p, ph, abortp);   // the pass has read A and written dZ
        if (more) bulk_g2s(sA, next + kTileA, kSq, bar_in);
        bulk_s2g(step_tiles(p, I, K) + kTileA, sZ, kSq);   // behind the loads, which would queue behind it
        bulk_commit();
        if (more) {
          mbar_wait_lazy_abort(bar_k, ph, abortp);
          load_qu(K + 1);
        }
        bulk_wait_read0();
        mbar_arrive(bar_zf);
      }
    }
    __syncwarp();
  } else {
  const uint32_t aVu = smem_u32(sVu), aT = smem_u32(sT), aA = smem_u32(sA), aS = smem_u32(sS), aG = smem_u32(sG), aQu = smem_u32(sQu),
                 aZ = smem_u32(sZ);
  // ---- the masked T = tril(Qc Vu^T)
  if (warp == 0 && elect_one()) {
    mbar_wait(bar_res, 0, abortp);
    tc_fence_after();
    gemm_kk_t<2>(tmem + C_DA, aZ, aVu, ID_KK, false);
    mma_commit(bar_t);
  }
  __syncwarp();
  mbar_wait(bar_t, 0, abortp);
  tc_fence_after();
  {
    float v[32];
    tmem_ld32_lower(trow + C_DA + c0, row, c0, v);
    store_row32<T>(sT, kPanelB, row, c0, v);
  }
  sync_passes();
  for (int K = 0; K <= I; ++K) {
    const uint32_t ph = K & 1;
    // ---- dA/scale = Gb Vu^T + dSu^T T;  dvu += A^T Gb;  dT += dSu A
    if (warp == 0 && elect_one()) {
      B128_MARK(512, K, 0);
      mbar_wait(bar_in, ph, abortp);
      tc_fence_after();
      B128_MARK(512, K, 1);
      if (!last) {
        gemm_kk_t<2>(tmem + C_DA, aG, aVu, ID_KK, false);
        gemm_mm_t<8>(tmem + C_DVU, aA, aG, ID_MM, K > 0);
        mma_commit(bar_g);
      }
      gemm_mm_t<8>(tmem + C_DA, aS, aT, ID_MM, !last);
      mma_commit(bar_da);
      gemm_km_t<8>(tmem + C_DT, aS, aA, ID_KM, K > 0);
      mma_commit(bar_v);
    }
    __syncwarp();
    B128_MARK(512, K, 2);
    mbar_wait(bar_da, ph, abortp);   // (dZ's last reader, the dku product, came before these)
    if (K > 0) mbar_wait(bar_zf, ph ^ 1, abortp);   // and its copy has been made
    tc_fence_after();
    B128_MARK(512, K, 3);
    {
      float v[32], a[32];
      tmem_ld32(trow + C_DA + c0, v);
      load_row32<T>(sA, kPanelB, row, c0, a);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; j += 2) {
        const float2 g = make_float2(a[j], a[j + 1]);
        const float2 x = mul2(mul2(make_float2(v[j], v[j + 1]), splat(p.scale)), fma2(mul2(g, splat(-1.f)), g, g));   // a (1 - a) = a - a a
        v[j] = x.x; v[j + 1] = x.y;
      }
      store_row32<T>(sZ, kPanelB, row, c0, v);
    }
    sync_passes();
    B128_MARK(512, K, 4);
    // ---- dku += dZ^T Qu
    if (warp == 0 && elect_one()) {
      mbar_wait(bar_qu, ph, abortp);
      B128_MARK(512, K, 5);
      tc_fence_after();
      gemm_mm_t<8>(tmem + C_DKU, aZ, aQu, ID_MM, K > 0);
      mma_commit(bar_k);
    }
    if (warp == 1 && elect_one()) mbar_arrive(bar_p);
    __syncwarp();
  }
  // ---- the masked dT (over dZ):  dvu += dT^T Qc;  dqc += dT Vu
  mbar_wait(bar_zf, (uint32_t)I & 1u, abortp);
  mbar_wait(bar_k, (uint32_t)I & 1u, abortp);
  tc_fence_after();
  if (warp == 4 && elect_one()) {
    mbar_expect_tx(bar_res, kSq);
    load_op(sQu, m_qc, bar_res, i0, h, b);
  }
  __syncwarp();
  {
    float v[32];
    tmem_ld32_lower(trow + C_DT + c0, row, c0, v);
    store_row32<T>(sZ, kPanelB, row, c0, v);
  }
  sync_passes();
  if (warp == 0 && elect_one()) {
    mbar_wait(bar_res, 1, abortp);
    tc_fence_after();
    gemm_mm_t<8>(tmem + C_DVU, aZ, aQu, ID_MM, !last);
    gemm_km_t<8>(tmem + C_DA, aZ, aVu, ID_KM, false);
    mma_commit(bar_da);
  }
  __syncwarp();
  const int irow = i0 + row;
  float v[32];
  tmem_ld32(trow + C_DKU + c0, v);
  tmem_ld_wait();
  if (irow < p.N) store_grad32<T>(grad_row<T>(p.dku, b, h, irow, c0), v, p.scale);
  mbar_wait(bar_da, (uint32_t)(I + 1) & 1u, abortp);
  tc_fence_after();
  tmem_ld32(trow + C_DVU + c0, v);
  tmem_ld_wait();
  if (irow < p.N) store_grad32<T>(grad_row<T>(p.dvu, b, h, irow, c0), v, p.scale);
  tmem_ld32(trow + C_DA + c0, v);
  tmem_ld_wait();
  if (irow < p.N) {
    const float4* acc = reinterpret_cast<const float4*>(p.acc_dqc + ((int64_t)bh * p.N + irow) * 128 + c0);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 q = acc[j];
      v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
    }
    store_grad32<T>(grad_row<T>(p.dqc, b, h, irow, c0), v, p.scale);
  }
  }
  B128_END(512)
}

// ------------------------------------------------------------------------------------------------ dqu
// A stream of dZ and Ku tiles through three stages into one accumulator.
template <typename T>
__global__ void __launch_bounds__(128)
castle_bwd128_dqu_kernel(const BwdParams p, const __grid_constant__ CUtensorMap m_ku) {
  constexpr uint32_t ID_KM = make_idesc(128, 128, Elem<T>::fmt, false, true, false);
  const int K = blockIdx.y, k0 = K * kBlkB, steps = p.nblk - K;
  B128_BEGIN(6 * kSq, 7, 128)
  uint64_t *bar_in = bars, *bar_done = bars + 3, *bar_end = bars + 6;   // three, three, one
  if (warp == 0 && elect_one()) {
    auto load = [&](int n) {
      const int s = n % 3;
      mbar_expect_tx(bar_in + s, 2 * kSq);
      bulk_g2s(smem + s * 2 * kSq, step_tiles(p, K + n, K) + kTileA, kSq, bar_in + s);
      load_op(smem + (s * 2 + 1) * kSq, m_ku, bar_in + s, k0 + n * kBlkB, h, b);
    };
    for (int n = 0; n < steps && n < 3; ++n) load(n);
    for (int n = 0; n < steps; ++n) {
      const int s = n % 3;
      mbar_wait(bar_in + s, (uint32_t)(n / 3) & 1u, abortp);
      tc_fence_after();
      gemm_km_t<8>(tmem, smem_u32(smem + s * 2 * kSq), smem_u32(smem + (s * 2 + 1) * kSq), ID_KM, n > 0);
      mma_commit(bar_done + s);
      if (n > 0 && n + 2 < steps) {   // the stage of the step before: its product is done or about to be
        mbar_wait(bar_done + (n - 1) % 3, (uint32_t)((n - 1) / 3) & 1u, abortp);
        load(n + 2);
      }
    }
    mma_commit(bar_end);
  }
  __syncwarp();
  mbar_wait(bar_end, 0, abortp);
  tc_fence_after();
  const int krow = k0 + tid;
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    float v[32];
    tmem_ld32(trow + c * 32, v);
    tmem_ld_wait();
    if (krow < p.N) store_grad32<T>(grad_row<T>(p.dqu, b, h, krow, c * 32), v, p.scale);
  }
  (void)lane;
  B128_END(128)
}

// ------------------------------------------------------------------------------------------------ launches
constexpr int kKvSplitMin = 7;   // shorter walks are not cut
constexpr int64_t kTileScratchLimit = (int64_t)8 << 30;
size_t bwd128_pair_bytes(int nblk) { return (size_t)nblk * (nblk + 1) / 2 * kStepTiles; }
int bwd128_chunk_pairs(int BH, int nblk) {
  int64_t n = kTileScratchLimit / (int64_t)bwd128_pair_bytes(nblk);
  if (n < 1) n = 1;
  return (int)(n < BH ? n : BH);
}

template <typename T>
static int launch_bwd128_t(const BwdParams& p, const CUtensorMap* in, cudaStream_t st) {
  constexpr int D = 128;
  const void* kernels[5] = {(const void*)castle_bwd128_kv_kernel<T, false>, (const void*)castle_bwd128_reverse_kernel<T>,
                            (const void*)castle_bwd128_la_kernel<T>, (const void*)castle_bwd128_dqu_kernel<T>, (const void*)castle_bwd128_kv_kernel<T, true>};
  const size_t smem[5] = {kB128Smem, 6 * kSq + 256, kB128Smem, 6 * kSq + 256, kB128Smem};
  for (int i = 0; i < 5; ++i) {
    cudaError_t e = cudaFuncSetAttribute(kernels[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem[i]);
    if (e != cudaSuccess) return cuda_fail(e, "castle_bwd attribute");
  }
  CUtensorMap acc;
  int rc = make_tmap_f32_rows(&acc, p.acc_dqc, p.B * p.H, p.N, D, "gradient workspace");
  if (rc) return rc;
  const int64_t rows = (int64_t)p.B * p.H * p.N;
  constexpr int RPB = 256 / (D / 8);
  castle_bwd_delta_kernel<T, D, 1><<<(unsigned)((rows + RPB - 1) / RPB), 256, 0, st>>>(p);
  const int BH = p.B * p.H, chunk = p.chunk_pairs;
  ev_start(CASTLE_KERNEL_BWD, st);
  for (int bh0 = 0; bh0 < BH; bh0 += chunk) {
    BwdParams q = p;
    q.bh0 = bh0;
    q.ntiles = (int64_t)p.nblk * (p.nblk + 1) / 2;
    const int pairs = BH - bh0 < chunk ? BH - bh0 : chunk;
    // Key blocks whose walks are cut: the longer half, where the steps per SM are less than half the longest walk.  us of forward and
    // backward, uncut / cut: 4 pairs x 4096 positions 535 / 480 (0.45), 8 x 2048 301 / 287 (0.46), 10 x 1024 163 / 157 (0.30),
    // 12 x 1500 247 / 248 (0.53); above that the repeated state costs more than the balance gains: 16 x 1333 248 / 263 (0.65), 8 x
    // 3000 469 / 480 (0.68).
    const float load = (float)pairs * (float)(p.nblk + 1) * (0.5f / 148.f);
    q.kv_split = p.nblk >= kKvSplitMin && load < 0.5f ? std::max(0, std::min(p.nblk + 1 - kKvSplitMin, p.N / (2 * kBlkB))) : 0;
    const dim3 grid(pairs, p.nblk), kv_grid(pairs, q.kv_split ? 2 * p.nblk : p.nblk);
    // in[]: qc, kc, vc, qu, ku, vu, dout
    // each starts while the one before it ends
    cudaError_t e = launch_kernel(q.kv_split ? castle_bwd128_kv_kernel<T, true> : castle_bwd128_kv_kernel<T, false>, kv_grid, kSplitThreads, smem[0], st, true, q, in[0], in[1], in[2], in[3], in[4], in[5], in[6], acc);
    if (e == cudaSuccess && p.nblk > 1) e = launch_kernel(castle_bwd128_reverse_kernel<T>, dim3(pairs, p.nblk - 1), kB128Threads, smem[1], st, true, q, in[0]);
    if (e == cudaSuccess) e = launch_kernel(castle_bwd128_la_kernel<T>, grid, kB128Threads + 32, smem[2], st, true, q, in[0], in[3], in[5]);
    if (e == cudaSuccess) e = launch_kernel(castle_bwd128_dqu_kernel<T>, grid, 128, smem[3], st, true, q, in[4]);
    if (e == cudaSuccess && q.kv_split)
      e = launch_kernel(castle_bwd128_parts_kernel<T>, dim3(pairs, q.kv_split, kBlkB / 16), 256, 0, st, true, q);
    if (e != cudaSuccess) return cuda_fail(e, "castle_bwd launch");
  }
  ev_stop(CASTLE_KERNEL_BWD, st);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_bwd launch");
}

int launch_bwd128(const BwdParams& p, int dtype, const CUtensorMap* in_maps, cudaStream_t st) {
  return dtype == CASTLE_BF16 ? launch_bwd128_t<__nv_bfloat16>(p, in_maps, st) : launch_bwd128_t<__half>(p, in_maps, st);
}

}  // namespace castle
