// CASTLE parallel backward for sm_100a (dim_head 64).
//
// One CTA owns a block K of 128 keys and walks the query blocks I from the last
// one DOWN to K, recomputing the scores flash-style.  Two 128 x d fp32 states
// live in tensor memory for the whole walk:
//   W_K  the forward's lookahead state.  It starts as the forward's final state
//        (= U[K], saved unrounded) and block I is peeled off with a negated
//        product, W_K -= A[K,I] @ Vu[I], so that before the scores of block I
//        are rebuilt it equals what the forward saw there.
//   G_K  = sum_{I' > I} dSu[I',K]^T @ Qc[I']: everything later queries
//        contribute to d(loss)/d(W_K); it yields dA and dvu for block I.
// dkc, dvc and dqu of the key block accumulate in tensor memory as well and are
// written once at the end.  The gradients indexed by the query/position block
// (dqc, dvu, dku) are summed over key blocks with TMA reduce-adds (fp32) into a
// workspace that a last kernel scales and casts.  A thread owns 32 consecutive
// columns of one accumulator row; the soft-max statistics (lse, delta) of its
// row sit in registers.
//
// Shared memory (224 KB) is time-shared: the 128x128 16-bit operands the
// threads produce (gate A, masked T, P, dS, dSu, dZ, dT) rotate through four
// 32 KB slots, two of which overlay input tiles that are dead by then.
//
// What bounds a step: some 1.5 MB through shared memory (11.7 k cycles at 128 bytes a cycle) and a chain of nine products
// with a pass behind each.  So sixteen warps do the passes and nothing else, one warp issues every product and one moves the
// tiles: a thread that issues products waits as long as the tensor unit's queue is full, and its warp then came late to the
// pass that everybody waited for.  A pass reports twice, on named barriers where only the issuing warp waits: when the accumulator
// columns are in registers (the next product into them starts under the arithmetic) and when its results are in shared memory.
// Step 19.1 k -> 15.5 k cycles; the kernel at B=4 N=4096 H=16 2390 -> 1936 us, B=16 H=8 N=1024 387 -> 332, 15 pairs of 777 78.2 -> 63.3.
// The first tiles and the state are asked for before the CTA's first barrier: whole backward of 1024 pairs of one block 169.2 ->
// 167.5 us, B=16 H=8 N=1024 370 -> 367.5.  That a CTA leaves when its last reduces have been read, not done, makes no difference to either.
#include "bwd_common.cuh"

namespace castle {

// Optional phase timing (debug builds only): thread 0 of CTA (0,0) stores clock64() at each phase
// boundary of its first steps behind the fp32 workspace, which the host dumps; behind 8 x 32 of these the warp that issues
// the products does, when what an event let it issue is on its way (none for kEvDz, which lets it issue nothing).
#ifdef CASTLE_PHASE_TIMING
#define BISSUE_MARK(k) do { if (lane == 0 && blockIdx.x == 0 && blockIdx.y == 0 && n < 8) p.timing[256 + n * 32 + (k)] = clock64(); } while (0)
#define BPHASE_MARK(i) do { if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && n < 8) p.timing[n * 32 + (i)] = clock64(); } while (0)
#else
#define BPHASE_MARK(i) do { } while (0)
#define BISSUE_MARK(k) do { } while (0)
#endif

// Timing experiments only (never in the shipped library): drop the reduces to see what they cost.
#ifdef CASTLE_TIMING_SKIP_REDUCE
#define tma_reduce_add_3d(...) do { } while (0)
#endif

// The events of a step that the issuing warp takes (ev_arrive), in their order; they take turns on four named barriers.
enum BwdEvent { kEvReadZ, kEvGate, kEvT, kEvCopyW, kEvReadSu, kEvReadSc, kEvP, kEvReadDp, kEvDs, kEvReadDa, kEvDz, kEvReadDt, kEvDt, kEvReadX, kEvCount };
__device__ constexpr int bwd_event(int k) { return 1 + k % 4; }
// Those that the moving warp takes, and after each other step by step.
enum BwdStaged { kEvDqc = 5, kEvDku = 6, kEvDvu = 7 };   // and 8 to 10 in odd steps
constexpr int kWorkers = 11, kEpilogue = 12;             // of the passes among themselves: all 512, and 12 to 14 a chunk group each

template <typename T, int D>
__global__ void __launch_bounds__(kSplitThreads, 1)
castle_bwd_kernel(const BwdParams p, const __grid_constant__ CUtensorMap m_qc, const __grid_constant__ CUtensorMap m_kc,
                  const __grid_constant__ CUtensorMap m_vc, const __grid_constant__ CUtensorMap m_qu,
                  const __grid_constant__ CUtensorMap m_ku, const __grid_constant__ CUtensorMap m_vu,
                  const __grid_constant__ CUtensorMap m_do, const __grid_constant__ CUtensorMap m_acc_dqc,
                  const __grid_constant__ CUtensorMap m_acc_dvu, const __grid_constant__ CUtensorMap m_acc_dku) {
  static_assert(D == 64, "this kernel is laid out for dim_head 64");
  constexpr uint32_t OPB = kPanelB;          // one d-wide operand tile (16 KB)
  constexpr uint32_t SQB = 2 * kPanelB;      // one 128x128 tile (32 KB)
  constexpr int FMT = Elem<T>::fmt;
  constexpr uint32_t ID_SQ_KK = make_idesc(128, 128, FMT, false, false, false);
  constexpr uint32_t ID_SQ_KM = make_idesc(128, 128, FMT, false, true, false);
  constexpr uint32_t ID_SQ_MM = make_idesc(128, 128, FMT, true, true, false);
  constexpr uint32_t ID_D_KM = make_idesc(128, D, FMT, false, true, false);
  constexpr uint32_t ID_D_KM_NEG = make_idesc(128, D, FMT, false, true, true);
  constexpr uint32_t ID_D_MM = make_idesc(128, D, FMT, true, true, false);
  constexpr float kLog2e = 1.4426950408889634f;
  // tensor-memory columns
  constexpr uint32_t C_W = 0, C_G = 64, C_DKC = 128, C_DVC = 192, C_DQU = 256, C_S = 320, C_X = 448;
  constexpr uint32_t C_X2 = C_S, C_X3 = C_S + 64;

  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQu = smem;                 // resident
  uint8_t* sKc = sQu + OPB;            // resident
  uint8_t* sQc = sKc + OPB;            // per step
  uint8_t* sVu = sQc + OPB;            // per step
  uint8_t* sVD = sVu + OPB;            // [Vc | dO] per step, later slot 3: dS -> dT -> staging of dvu
  uint8_t* sVc = sVD;
  uint8_t* sdO = sVD + OPB;
  uint8_t* sKP = sVD + SQB;            // [Ku | spare], later slot 4: P -> dSu, then the next Ku in the first half
  uint8_t* sWb = sKP + SQB;            // copy of W, then Ku again
  uint8_t* sGb = sWb + OPB;
  uint8_t* sA = sGb + OPB;             // slot 1: gate A
  uint8_t* sT = sA + SQB;              // slot 2: masked T -> dZ -> staging of dku
  // Each of these completes once per step.
  __shared__ uint64_t bar_res, bar_load, bar_vd, bar_ku, bar_kn;   // tiles
  __shared__ uint64_t bar_z, bar_t, bar_w, bar_su, bar_sc, bar_dp, bar_dv, bar_da, bar_dt, bar_g, bar_x, bar_l;   // products
  __shared__ uint64_t bar_end;                                     // once: no product is in flight
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_flag;
  __shared__ float zero_s;

  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int bh = blockIdx.x, K = blockIdx.y;
  const int b = bh / p.H, h = bh % p.H;
  const int k0 = K * kBlkB, walk = p.nblk - K;

  // The first tiles are on their way before the barrier below; nothing in flight writes what they read (only the sums and delta are
  // being written by the kernel before this one).
  if (warp == 17 && elect_one()) {
    if (smem_u32(smem) & 1023u) atomicOr(p.status, CASTLE_STATUS_BAD_LAUNCH);
    uint64_t* const bars[18] = {&bar_res, &bar_load, &bar_vd, &bar_ku, &bar_kn, &bar_z, &bar_t, &bar_w, &bar_su,
                                &bar_sc, &bar_dp, &bar_dv, &bar_da, &bar_dt, &bar_g, &bar_x, &bar_l, &bar_end};
#pragma unroll
    for (int i = 0; i < 18; ++i) mbar_init(bars[i], bars[i] == &bar_t || bars[i] == &bar_w ? 2 : 1);   // these two: the product, and the slot written next is free
    mbar_fence_init();
    abort_flag = 0;
    zero_s = 0.f;
    const int il = (p.nblk - 1) * kBlkB;
    mbar_expect_tx(&bar_res, 2 * OPB);
    tma_load_4d(sQu, &m_qu, &bar_res, 0, k0, h, b);
    mbar_expect_tx(&bar_kn, OPB);
    tma_load_4d(sKP, &m_ku, &bar_kn, 0, il, h, b);
    tma_load_4d(sKc, &m_kc, &bar_res, 0, k0, h, b);
    mbar_expect_tx(&bar_load, 2 * OPB);
    tma_load_4d(sQc, &m_qc, &bar_load, 0, il, h, b);
    tma_load_4d(sVu, &m_vu, &bar_load, 0, il, h, b);
    mbar_arrive(&bar_t);
    mbar_arrive(&bar_w);
    mbar_expect_tx(&bar_vd, 2 * OPB);
    tma_load_4d(sVc, &m_vc, &bar_vd, 0, k0, h, b);
    tma_load_4d(sdO, &m_do, &bar_vd, 0, il, h, b);
  }
  __syncwarp();
  constexpr int kWLoads = kBlkB * (D / 4) / kSplitWorkers;
  float4 w0[kWLoads];   // of the forward's final state
  if (warp < kSplitWorkers / 32) {
#pragma unroll
    for (int i = 0; i < kWLoads; ++i) {
      const int e = i * kSplitWorkers + tid, r = e / (D / 4), c = e % (D / 4);
      w0[i] = (k0 + r < p.N) ? *reinterpret_cast<const float4*>(p.w_state + ((int64_t)bh * p.N + k0 + r) * D + c * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  if (warp == 0) { tmem_alloc(&tmem_base_s, 512); tmem_relinquish(); }
  overlap_wait();   // launched while delta is being written
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_s;
  volatile int* abortp = &abort_flag;

  if (warp >= kSplitWorkers / 32) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(SplitRegs<T>::others));
    if (warp == 16) {
      // ---- the products, in the order that the passes need them; what a pass does not wait for goes behind its commit
      // operand addresses are made where they are used: kept in registers over the step they would be spilled
      auto at = [&](const uint8_t* tile) {
        uint32_t base = smem_u32(smem);
        asm volatile("" : "+r"(base));
        return base + (uint32_t)(tile - smem);
      };
      auto next = [&](int k) {
        __syncwarp();
        ev_wait(bwd_event(k), kSplitWorkers);
        tc_fence_after();
      };
      auto issue_z = [&](uint32_t ph) {
        mbar_wait(&bar_kn, ph, abortp);
        tc_fence_after();
        gemm_kk_t<1>(tmem + C_S, at(sQu), at(sKP), ID_SQ_KK, false);
        mma_commit(&bar_z);
      };
      if (elect_one()) {
        mbar_wait(&bar_res, 0, abortp);
        issue_z(0);
      }
#pragma unroll 1
      for (int n = 0; n < walk; ++n) {
        const uint32_t ph = n & 1;
        const bool first = n == 0, diag = n == walk - 1;
        next(kEvReadZ);
        if (elect_one()) {
          mbar_wait(&bar_load, ph, abortp);
          tc_fence_after();
          gemm_kk_t<1>(tmem + C_S, at(sQc), at(sVu), ID_SQ_KK, false);          // T = Qc[I] Vu[I]^T, while the gate is formed
          mma_commit(&bar_t);
        }
        BISSUE_MARK(kEvReadZ);
        next(kEvGate);
        if (elect_one()) {
          if (!diag) gemm_km_t<8>(tmem + C_W, at(sA), at(sVu), ID_D_KM_NEG, true);   // W_K -= A Vu[I], while T is masked; zero at the diagonal block, where nothing reads it
          mma_commit(&bar_w);
        }
        BISSUE_MARK(kEvGate);
        next(kEvT);        // masked
        if (elect_one()) gemm_kk_t<2>(tmem + C_S, at(sT), at(sA), ID_SQ_KK, false);    // Su/scale = T A^T + Qc[I] Wb^T, while W is copied
        BISSUE_MARK(kEvT);
        next(kEvCopyW);
        if (elect_one()) {
          if (!diag) gemm_kk_t<1>(tmem + C_S, at(sQc), at(sWb), ID_SQ_KK, true);
          mma_commit(&bar_su);
        }
        BISSUE_MARK(kEvCopyW);
        next(kEvReadSu);
        if (elect_one()) {
          gemm_kk_t<1>(tmem + C_S, at(sQc), at(sKc), ID_SQ_KK, false);          // Sc/scale = Qc[I] Kc[K]^T, while silu' is formed
          mma_commit(&bar_sc);
        }
        BISSUE_MARK(kEvReadSu);
        next(kEvReadSc);
        if (elect_one()) {
          mbar_wait(&bar_vd, ph, abortp);
          tc_fence_after();
          gemm_kk_t<1>(tmem + C_S, at(sdO), at(sVc), ID_SQ_KK, false);          // dP = dO[I] Vc[K]^T, while P is formed
          mma_commit(&bar_dp);
        }
        BISSUE_MARK(kEvReadSc);
        next(kEvP);
        if (elect_one()) {
          gemm_mm_t<8>(tmem + C_DVC, at(sKP), at(sdO), ID_D_MM, !first);        // dvc += P^T dO[I], while dS is formed
          mma_commit(&bar_dv);
        }
        BISSUE_MARK(kEvP);
        next(kEvReadDp);
        if (!first && elect_one()) gemm_kk_t<1>(tmem + C_S, at(sGb), at(sVu), ID_SQ_KK, false);   // dA/scale = Gb Vu[I]^T + dSu^T T
        BISSUE_MARK(kEvReadDp);
        next(kEvDs);       // and dSu
        if (elect_one()) {
          gemm_mm_t<8>(tmem + C_S, at(sKP), at(sT), ID_SQ_MM, !first);
          mma_commit(&bar_da);
          gemm_mm_t<8>(tmem + C_DKC, at(sVD), at(sQc), ID_D_MM, !first);        // dkc += dS^T Qc[I]
          gemm_km_t<8>(tmem + C_X, at(sVD), at(sKc), ID_D_KM, false);           // X = dS Kc[K] + dSu Wb + dT Vu[I]
        }
        BISSUE_MARK(kEvDs);
        next(kEvReadDa);
        if (elect_one()) {
          gemm_km_t<8>(tmem + C_S, at(sKP), at(sA), ID_SQ_KM, false);           // dT = dSu A, while dZ is formed
          mma_commit(&bar_dt);
          if (!diag) {
            gemm_km_t<8>(tmem + C_X, at(sKP), at(sWb), ID_D_KM, true);
            gemm_mm_t<8>(tmem + C_G, at(sKP), at(sQc), ID_D_MM, !first);        // G += dSu^T Qc[I]
          }
          mma_commit(&bar_g);
        }
        BISSUE_MARK(kEvReadDa);
        next(kEvDz);
        next(kEvReadDt);
        if (elect_one()) gemm_mm_t<8>(tmem + C_X3, at(sT), at(sQu), ID_D_MM, false);   // X3 = dZ^T Qu[K]
        BISSUE_MARK(kEvReadDt);
        next(kEvDt);       // masked
        if (elect_one()) {
          gemm_mm_t<8>(tmem + C_X2, at(sVD), at(sQc), ID_D_MM, false);          // X2 = dT^T Qc[I] + A^T Gb
          gemm_km_t<8>(tmem + C_X, at(sVD), at(sVu), ID_D_KM, true);
          mbar_wait(&bar_ku, ph, abortp);
          tc_fence_after();
          gemm_km_t<8>(tmem + C_DQU, at(sT), at(sWb), ID_D_KM, !first);         // dqu += dZ Ku[I]
          mma_commit(&bar_x);
          if (!first) gemm_mm_t<8>(tmem + C_X2, at(sA), at(sGb), ID_D_MM, true);
          mma_commit(&bar_l);
        }
        BISSUE_MARK(kEvDt);
        next(kEvReadX);
        if (!diag && elect_one()) issue_z(ph ^ 1);
        BISSUE_MARK(kEvReadX);
      }
      __syncwarp();
      if (elect_one()) {
        mma_commit(&bar_end);
        mbar_drain(&bar_end, 0);
      }
      __syncwarp();
    } else if (warp == 17) {
      // ---- the tiles.  The TMA unit works its queue off in order and a reduce takes thousands of cycles, so loads go ahead of them.
      int n = 0;
      bool half = false;   // a wait that did not end well ended the walk, the second of its step
#pragma unroll 1
      for (; n < walk; ++n) {
        const uint32_t ph = n & 1;
        const bool more = n + 1 < walk;
        const int i0 = (p.nblk - 1 - n) * kBlkB, in0 = i0 - kBlkB, odd = 3 * (n & 1);
        if (mbar_wait_failed(&bar_g, ph, abortp)) break;                  // copy of W and dSu have been read
        if (elect_one()) {
          mbar_expect_tx(&bar_ku, OPB);
          tma_load_4d(sWb, &m_ku, &bar_ku, 0, i0, h, b);
          if (more) {
            mbar_expect_tx(&bar_kn, OPB);
            tma_load_4d(sKP, &m_ku, &bar_kn, 0, in0, h, b);
          }
        }
        __syncwarp();
        if (mbar_wait_failed(&bar_x, ph, abortp)) { half = true; break; } // Qc[I], Vu[I], Ku[I] as well
        if (more && elect_one()) {
          mbar_expect_tx(&bar_load, 2 * OPB);
          tma_load_4d(sQc, &m_qc, &bar_load, 0, in0, h, b);
          tma_load_4d(sVu, &m_vu, &bar_load, 0, in0, h, b);
        }
        __syncwarp();
        ev_wait(kEvDku + odd, 128);              // its slot is needed first
        if (elect_one()) {
          tma_reduce_add_3d(&m_acc_dku, sT, 0, i0, bh);
          tma_reduce_add_3d(&m_acc_dku, sT + kPanelB, 32, i0, bh);
          bulk_commit();
        }
        __syncwarp();
        ev_wait(kEvDqc + odd, 128);
        if (elect_one()) {
          tma_reduce_add_3d(&m_acc_dqc, sWb, 0, i0, bh);
          tma_reduce_add_3d(&m_acc_dqc, sKP + kPanelB, 32, i0, bh);
          bulk_commit();
        }
        __syncwarp();
        ev_wait(kEvDvu + odd, 256);
        if (elect_one()) {
          tma_reduce_add_3d(&m_acc_dvu, sVD, 0, i0, bh);
          tma_reduce_add_3d(&m_acc_dvu, sVD + kPanelB, 32, i0, bh);
          bulk_commit();
          bulk_wait_read2();
          if (more) mbar_arrive(&bar_t);         // T may go over the staging of dku
          bulk_wait_read1();
          if (more) mbar_arrive(&bar_w);         // and the copy of W and P over that of dqc
          bulk_wait_read0();
          if (more) {
            mbar_expect_tx(&bar_vd, 2 * OPB);
            tma_load_4d(sVc, &m_vc, &bar_vd, 0, k0, h, b);
            tma_load_4d(sdO, &m_do, &bar_vd, 0, in0, h, b);
          }
        }
        __syncwarp();
      }
      if (elect_one()) {
        if (*abortp) {   // tiles that were asked for and that nobody may have waited for must not land after the CTA has left
          const int last = n < walk ? n : walk - 1;
          mbar_drain(&bar_res, 0);
          mbar_drain(&bar_load, last & 1);
          mbar_drain(&bar_vd, last & 1);
          mbar_drain(&bar_ku, (n == walk || half ? last : last - 1) & 1);
          mbar_drain(&bar_kn, (half && last + 1 < walk ? last + 1 : last) & 1);
        }
        bulk_wait_read0();   // the sums themselves are complete when the kernel is
      }
      __syncwarp();
      for (; n < walk; ++n) {   // nothing is asked for any more, for a barrier's last phase may still be open
        const int odd = 3 * (n & 1);
        ev_wait(kEvDku + odd, 128);
        ev_wait(kEvDqc + odd, 128);
        ev_wait(kEvDvu + odd, 256);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(SplitRegs<T>::passes));
    const int quarter = warp & 3, cc = warp >> 2;
    const int row = quarter * 32 + lane;
    const int c0 = cc * 32;
    const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16);
    const float sl2 = p.scale * kLog2e, half_scale = 0.5f * p.scale;
    bool failed;
    auto wait = [&](uint64_t* bar, uint32_t ph) {
      failed = mbar_wait_failed(bar, ph, abortp);   // (one polling lane a warp: 1970 -> 2126 us at B=4 N=4096 H=16)
      tc_fence_after();
    };
    // a wait that did not end well ends the walk; `arrived`: the events of this step that the warp has arrived on before
#define BWD_CHECK(ARRIVED) if (failed) { arrived = ARRIVED; goto stopped; }
    auto read = [&](int k) { return ev_arrive_read(bwd_event(k), kSplitWorkers, &zero_s); };
    auto stored = [&](int k) {
      fence_async_smem();
      tc_fence_before();
      ev_arrive(bwd_event(k), kSplitWorkers);
    };
    int n = 0;
    uint32_t arrived = 0;
    // W_K starts as the forward's final state, brought in whole lines (rows of 64 floats over the threads, through the gate's slot):
    // a row per lane, here and where the gradients are stored, took 2 us of a key block each; 1036 pairs of one block 150.5 ->
    // 142.3 us, B=16 H=8 N=1024 402 -> 392 us
#pragma unroll
    for (int i = 0; i < kWLoads; ++i) {
      const int e = i * kSplitWorkers + tid, r = e / (D / 4), c = e % (D / 4);
      *reinterpret_cast<float4*>(sA + (c >> 3) * kPanelB + swz_off(r, c & 7)) = w0[i];
    }
    asm volatile("bar.sync %0, %1;" ::"n"(kWorkers), "n"(kSplitWorkers) : "memory");
    if (c0 < D) {
      float v[32];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 q = *reinterpret_cast<const float4*>(sA + cc * kPanelB + swz_off(row, j));
        v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
      }
      tmem_st32(trow + C_W + c0, v);
      tmem_st_wait();
    }
    asm volatile("bar.sync %0, %1;" ::"n"(kWorkers), "n"(kSplitWorkers) : "memory");

#pragma unroll 1
    for (; n < walk; ++n) {
      const uint32_t ph = n & 1;
      const int I = p.nblk - 1 - n, irow = I * kBlkB + row;
      const bool diag = I == K, rvalid = irow < p.N;
      BPHASE_MARK(0);
      wait(&bar_z, ph);
      BPHASE_MARK(1);
      {  // gate A (rows k, columns j), zero unless j > k
        float v[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        BWD_CHECK(kEvReadZ)
        const float hs = half_scale + read(kEvReadZ);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 a = sigmoid2(make_float2(v[j], v[j + 1]), hs);
          v[j] = a.x; v[j + 1] = a.y;
        }
        if (diag) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = (c0 + j > row) ? v[j] : 0.f;
        }
        store_row32<T>(sA, kPanelB, row, c0, v);
      }
      stored(kEvGate);
      BPHASE_MARK(2);
      wait(&bar_t, ph);
      BPHASE_MARK(3);
      {  // masked T (rows i, columns j <= i), unscaled
        float v[32];
        tmem_ld32_lower(trow + C_S + c0, row, c0, v);
        BWD_CHECK(kEvT)
        store_row32<T>(sT, kPanelB, row, c0, v);
      }
      stored(kEvT);
      wait(&bar_w, ph);
      BWD_CHECK(kEvCopyW)
      BPHASE_MARK(4);
      if (c0 < D) {  // 16-bit copy of the peeled state
        float v[32];
        tmem_ld32(trow + C_W + c0, v);
        tmem_ld_wait();
        store_row32<T>(sWb, kPanelB, row, c0, v);
      }
      stored(kEvCopyW);
      BPHASE_MARK(5);
      // loaded here, not at the top of the step, where the wait for Z is short
      const float lse_i = rvalid ? p.lse[(int64_t)bh * p.N + irow] : 0.f, delta_i = rvalid ? p.delta[(int64_t)bh * p.N + irow] : 0.f;
      wait(&bar_su, ph);
      BPHASE_MARK(6);
      uint32_t dpk[16];  // silu'(Su), two 16-bit values per register
      uint32_t ppk[16];  // P
      {
        float v[32], w[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        BWD_CHECK(kEvReadSu)
        const float hs = half_scale + read(kEvReadSu);
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
        BPHASE_MARK(7);
        wait(&bar_sc, ph);
        BPHASE_MARK(8);
        // P = exp(S - lse) (rows i, columns k); into slot 4 over Ku
        tmem_ld32(trow + C_S + c0, w);
        tmem_ld_wait();
        BWD_CHECK(kEvReadSc)
        const float s2 = sl2 + read(kEvReadSc);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 x = fma2(add2(make_float2(w[j], w[j + 1]), make_float2(v[j], v[j + 1])), splat(s2), splat(-lse_i * kLog2e));
          const float2 e = j % 16 == 0 ? exp2_fma2(x) : make_float2(ex2_approx(x.x), ex2_approx(x.y));   // an eighth off the busiest unit
          v[j] = e.x; v[j + 1] = e.y;
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
        store_row32<T>(sKP, kPanelB, row, c0, v);
      }
      stored(kEvP);
      BPHASE_MARK(9);
      wait(&bar_dp, ph);
      BPHASE_MARK(10);
      {  // dS = P * (dP - delta) -> slot 3 (over Vc|dO); dSu = -dS * silu'(Su) -> slot 4 (over P)
        float v[32], w[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        BWD_CHECK(kEvReadDp)
        const float dl = delta_i + read(kEvReadDp);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 ds = mul2(Elem<T>::unpack2(ppk[j / 2]), add2(make_float2(v[j], v[j + 1]), splat(-dl)));
          const float2 du = mul2(ds, Elem<T>::unpack2(dpk[j / 2]));
          v[j] = ds.x; v[j + 1] = ds.y;
          w[j] = -du.x; w[j + 1] = -du.y;
        }
        wait(&bar_dv, ph);   // dO and P have been read
        BWD_CHECK(kEvDs)
        store_row32<T>(sVD, kPanelB, row, c0, v);
        store_row32<T>(sKP, kPanelB, row, c0, w);
      }
      stored(kEvDs);
      BPHASE_MARK(11);
      wait(&bar_da, ph);
      BPHASE_MARK(12);
      {  // dZ = dA * A * (1 - A) -> slot 2 (over T)
        float v[32], a[32];
        tmem_ld32(trow + C_S + c0, v);
        tmem_ld_wait();
        BWD_CHECK(kEvReadDa)
        const float sc = p.scale + read(kEvReadDa);
        load_row32<T>(sA, kPanelB, row, c0, a);
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          const float2 g = make_float2(a[j], a[j + 1]);
          const float2 x = mul2(mul2(make_float2(v[j], v[j + 1]), splat(sc)), fma2(mul2(g, splat(-1.f)), g, g));   // a (1 - a) = a - a a
          v[j] = x.x; v[j + 1] = x.y;
        }
        store_row32<T>(sT, kPanelB, row, c0, v);
      }
      stored(kEvDz);   // an event of its own: the wait below does not cover it
      BPHASE_MARK(13);
      wait(&bar_dt, ph);
      BPHASE_MARK(14);
      {  // masked dT (rows i, columns j <= i) -> slot 3 (over dS)
        float v[32];
        tmem_ld32_lower(trow + C_S + c0, row, c0, v);
        BWD_CHECK(kEvReadDt)
        read(kEvReadDt);
        store_row32<T>(sVD, kPanelB, row, c0, v);
      }
      stored(kEvDt);
      BPHASE_MARK(15);
      // The query block's gradients are staged as fp32 panels in operand slots that are dead by then and handed to TMA reduces
      // (whole lines at L2 instead of scattered atomics): chunk group 1 takes dqc (into the copy of W's slot and the spare half of
      // slot 4), group 2 dku (into slot 2), groups 0 and 3 a panel each of dvu (into slot 3).  Groups 1 and 2 also make the
      // 16-bit copy of G, including block I, for the next (lower) block; the next step's events order it.
      const int part = cc >> 1, staged = (cc == 1 ? kEvDqc : cc == 2 ? kEvDku : kEvDvu) + 3 * (n & 1);
      if (cc == 1 || cc == 2) {
        wait(&bar_x, ph);
        BWD_CHECK(kEvReadX)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float v[32];
          tmem_ld32(trow + (cc == 1 ? C_X : C_X3) + c * 32, v);
          tmem_ld_wait();
          if (c == 1) read(kEvReadX);
          store_row32_f32(cc == 2 ? sT + c * kPanelB : c == 0 ? sWb : sKP + kPanelB, row, v);
        }
        fence_async_smem();
        ev_arrive(staged, 128);
        wait(&bar_l, ph);
        BWD_CHECK(kEvCount + 1)
        if (!diag) {
          float v[32];
          tmem_ld32(trow + C_G + part * 32, v);
          tmem_ld_wait();
          store_row32<T>(sGb, kPanelB, row, part * 32, v);
        }
      } else {
        wait(&bar_l, ph);
        BPHASE_MARK(16);
        float v[32];
        tmem_ld32(trow + C_X2 + part * 32, v);
        tmem_ld_wait();
        BWD_CHECK(kEvReadX)
        read(kEvReadX);
        store_row32_f32(sVD + part * kPanelB, row, v);
        fence_async_smem();
        ev_arrive(staged, 256);
      }
      BPHASE_MARK(17);
    }
#undef BWD_CHECK
  stopped:
    for (; n < walk; ++n, arrived = 0) {   // what is left of the events
#pragma unroll 1
      for (; arrived < kEvCount; ++arrived) ev_wait(bwd_event((int)arrived), kSplitWorkers);
      if (arrived == kEvCount) ev_wait((cc == 1 ? kEvDqc : cc == 2 ? kEvDku : kEvDvu) + 3 * (n & 1), cc == 1 || cc == 2 ? 128 : 256);
    }

    // ---- key-block gradients: dkc (x scale), dvc, dqu (x scale); one chunk group each, through the gate's slot and the copy of
    // G, so that eight lanes store a row in whole lines
    if (cc < 3) {
      const uint32_t col = (cc == 0) ? C_DKC : (cc == 1 ? C_DVC : C_DQU);
      const castle_tensor_t& dt = (cc == 0) ? p.dkc : (cc == 1 ? p.dvc : p.dqu);
      const float mul = (cc == 1) ? 1.f : p.scale;
      uint8_t* panel = cc == 0 ? sA : (cc == 1 ? sA + kPanelB : sGb);
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        float v[32];
        tmem_ld32(trow + col + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] *= mul;
        store_row32<T>(panel, kPanelB, row, c * 32, v);
      }
      group_sync(kEpilogue + cc);
      T* dst = reinterpret_cast<T*>(dt.ptr) + b * dt.stride_b + h * dt.stride_h + (lane & 7) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int r = (quarter * 8 + j) * 4 + (lane >> 3);
        if (k0 + r < p.N)
          *reinterpret_cast<uint4*>(dst + (int64_t)(k0 + r) * dt.stride_n) = *reinterpret_cast<const uint4*>(panel + swz_off(r, lane & 7));
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
  if (tid == 0 && abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

template <typename T, int D>
static int launch_bwd(const BwdParams& p, const CUtensorMap* maps, cudaStream_t st) {
  constexpr size_t smem = 7 * kPanelB + 4 * 2 * kPanelB - kPanelB + 1024;  // 224 KB + alignment slack
  {  // per device, so set on every call (cheap)
    cudaError_t e = cudaFuncSetAttribute(castle_bwd_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_bwd attribute");
  }
  static std::atomic<bool> regs_known{false};
  if (const int rc = check_launch_regs(castle_bwd_kernel<T, D>, regs_known)) return rc;
  const int64_t rows = (int64_t)p.B * p.H * p.N;
  constexpr int RPB = 256 / (D / 8);
  castle_bwd_delta_kernel<T, D, 3><<<(unsigned)((rows + RPB - 1) / RPB), 256, 0, st>>>(p);
  dim3 grid(p.B * p.H, p.nblk);
  ev_start(CASTLE_KERNEL_BWD, st);
  cudaError_t e = launch_kernel(castle_bwd_kernel<T, D>, grid, kSplitThreads, smem, st, true, p, maps[0], maps[1], maps[2], maps[3], maps[4],
                                maps[5], maps[6], maps[7], maps[8], maps[9]);
  ev_stop(CASTLE_KERNEL_BWD, st);
  if (e == cudaSuccess) e = launch_kernel(castle_bwd_finish_kernel<T, D, 3>, dim3((unsigned)((rows + RPB - 1) / RPB)), 256, 0, st, true, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_bwd launch");
}

}  // namespace castle

using namespace castle;

// fp32 accumulators dqc, dvu, dku and delta; at dim_head 128, where only the first is summed into (the other two are
// reserved, so that the size a caller asks for does not depend on how the kernels share the work), rounded up so that
// the tile scratch behind them stays 1 KB aligned
static size_t bwd_acc_bytes(const castle_problem_t* p) {
  int64_t rows = (int64_t)p->batch * p->heads * p->seq_len;
  size_t b = (size_t)(rows * (3 * p->dim_head + 1) * sizeof(float));
  return p->dim_head == 128 ? (b + 1023) & ~(size_t)1023 : b;
}

extern "C" size_t castle_bwd_workspace_bytes(const castle_problem_t* p) {
  if (!p || p->seq_len <= 0 || p->batch <= 0 || p->heads <= 0) return 0;
  const int nblk = (p->seq_len + kBlkB - 1) / kBlkB;
  size_t tiles = p->dim_head == 128 ? (size_t)bwd128_chunk_pairs(p->batch * p->heads, nblk) * bwd128_pair_bytes(nblk) : 0;
  return bwd_acc_bytes(p) + tiles;
}

extern "C" int castle_bwd(const castle_problem_t* p, const castle_tensor_t* qc, const castle_tensor_t* kc,
                          const castle_tensor_t* vc, const castle_tensor_t* qu, const castle_tensor_t* ku,
                          const castle_tensor_t* vu, const castle_tensor_t* out, const castle_tensor_t* dout,
                          const float* lse, const float* w_state, const castle_tensor_t* dqc,
                          const castle_tensor_t* dkc, const castle_tensor_t* dvc, const castle_tensor_t* dqu,
                          const castle_tensor_t* dku, const castle_tensor_t* dvu, void* workspace,
                          size_t workspace_bytes, int32_t* status, void* stream) {
  if (!p) return reject("castle_bwd: null problem");
  if (p->batch <= 0 || p->heads <= 0 || p->seq_len <= 0) return reject("castle_bwd: empty problem");
  if (p->dim_head != 64 && p->dim_head != 128) return reject("castle_bwd: dim_head %d not supported (64 or 128)", p->dim_head);
  if (p->dtype != CASTLE_BF16 && p->dtype != CASTLE_F16) return reject("castle_bwd: dtype %d not supported (bf16, fp16)", p->dtype);
  int nblk = (p->seq_len + kBlkB - 1) / kBlkB;
  if (nblk > 65535) return reject("castle_bwd: sequence too long");
  int rc = 0;
  const castle_tensor_t* ts[14] = {qc, kc, vc, qu, ku, vu, dout, out, dqc, dkc, dvc, dqu, dku, dvu};
  const char* names[14] = {"qc", "kc", "vc", "qu", "ku", "vu", "dout", "out", "dqc", "dkc", "dvc", "dqu", "dku", "dvu"};
  for (int i = 0; i < 14; ++i)
    if (!tensor_ok(ts[i], p->dtype, names[i], &rc)) return rc;
  if (!lse || !w_state || !status) return reject("castle_bwd: lse, w_state and status must not be null");
  // dim_head 64: the accumulators.  dim_head 128: the accumulators and the tile hand-over scratch of at least
  // one (batch, head) pair; the pairs run in chunks of as many as the scratch the caller passed holds.
  const size_t need = castle_bwd_workspace_bytes(p), acc_bytes = bwd_acc_bytes(p);
  const size_t pair_bytes = p->dim_head == 128 ? bwd128_pair_bytes(nblk) : 0;
  const size_t least = p->dim_head == 128 ? acc_bytes + pair_bytes : need;
  if (!workspace || workspace_bytes < least)
    return reject("castle_bwd: workspace too small (%zu bytes; castle_bwd_workspace_bytes says %zu, the least that works is %zu)",
                  workspace_bytes, need, least);
  if (((uintptr_t)workspace) % 16) return reject("castle_bwd: workspace not 16-byte aligned");

  BwdParams bp;
  bp.B = p->batch; bp.H = p->heads; bp.N = p->seq_len; bp.nblk = nblk; bp.scale = p->scale;
  bp.lse = lse; bp.w_state = w_state;
  int64_t rows = (int64_t)p->batch * p->heads * p->seq_len;
  // dim_head 128: the tile hand-over scratch follows the accumulators
  bp.tiles = (uint8_t*)workspace + acc_bytes;
  bp.ntiles = 0; bp.bh0 = 0; bp.chunk_pairs = 0; bp.kv_split = 0;
  if (p->dim_head == 128) {
    size_t fit = (workspace_bytes - acc_bytes) / pair_bytes;
    bp.chunk_pairs = (int)(fit < (size_t)(p->batch * p->heads) ? fit : (size_t)(p->batch * p->heads));
  }
  bp.acc_dqc = (float*)workspace;
  bp.acc_dvu = bp.acc_dqc + rows * p->dim_head;
  bp.acc_dku = bp.acc_dvu + rows * p->dim_head;
  bp.delta = bp.acc_dku + rows * p->dim_head;
  bp.out = *out; bp.dout = *dout;
  bp.dqc = *dqc; bp.dkc = *dkc; bp.dvc = *dvc; bp.dqu = *dqu; bp.dku = *dku; bp.dvu = *dvu;
  bp.status = status;
#ifdef CASTLE_PHASE_TIMING
  bp.timing = (long long*)((char*)workspace + need);  // the caller leaves 8 KB beyond what castle_bwd_workspace_bytes asks for
  if (bp.chunk_pairs > bwd128_chunk_pairs(p->batch * p->heads, nblk)) bp.chunk_pairs = bwd128_chunk_pairs(p->batch * p->heads, nblk);
#endif
  CUtensorMap maps[10];
  for (int i = 0; i < 7; ++i) {
    rc = make_tmap_16bit(&maps[i], ts[i], p->dtype, p->batch, p->heads, p->seq_len, p->dim_head, kBlkB, names[i]);
    if (rc) return rc;
  }
  float* accs[3] = {bp.acc_dqc, bp.acc_dvu, bp.acc_dku};
  for (int i = 0; i < 3; ++i) {
    rc = make_tmap_f32_rows(&maps[7 + i], accs[i], p->batch * p->heads, p->seq_len, p->dim_head, "gradient workspace");
    if (rc) return rc;
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (p->dim_head == 128) return launch_bwd128(bp, p->dtype, maps, st);
  if (p->dtype == CASTLE_BF16) return launch_bwd<__nv_bfloat16, 64>(bp, maps, st);
  return launch_bwd<__half, 64>(bp, maps, st);
}
