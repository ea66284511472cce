// Shared by the backward kernels (dim_head 64 in bwd.cu, dim_head 128 in bwd128.cu): launch
// parameters, the delta pre-pass and the kernel that turns fp32 accumulators into gradients.
#pragma once
#include <atomic>
#include "common.cuh"
#include "sm100.cuh"

namespace castle {

constexpr int kBlkB = 128;
constexpr uint32_t kPanelB = kBlkB * 128;

struct BwdParams {
  int B, H, N, nblk;
  float scale;
  const float* lse;      // [BH][N]
  const float* w_state;  // [BH][N][D]
  float* delta;          // [BH][N]
  float* acc_dqc;        // [BH][N][D] fp32, zeroed
  float* acc_dvu;        // these two at dim_head 64
  float* acc_dku;
  uint8_t* tiles;        // dim_head 128: the tiles that its kernels hand on, per (pair, query block, key block)
  int64_t ntiles;        // query-block x key-block pairs per (batch, head) pair
  int bh0;               // dim_head 128: first (batch, head) pair of this launch (the pairs run in chunks)
  int chunk_pairs;       // dim_head 128: pairs per chunk (what the caller's scratch holds)
  int kv_split;          // dim_head 128: key blocks [0, kv_split) are walked in two parts; their sums use acc_dvu and acc_dku
  castle_tensor_t out, dout;
  castle_tensor_t dqc, dkc, dvc, dqu, dku, dvu;
  int32_t* status;
#ifdef CASTLE_PHASE_TIMING
  long long* timing;
#endif
};

// The kernels whose passes, products and tiles are the work of different warps (castle_bwd_kernel, castle_bwd128_kv_kernel): warps
// 0-15 do the passes, warp 16 issues the products, warp 17 moves tiles, two more fill up the warpgroup.  castle_bwd_kernel shares the
// launch's registers out anew, 640 x 96 = 61440 (SplitRegs).
constexpr int kSplitWorkers = 512, kSplitThreads = kSplitWorkers + 128;
constexpr int kSplitLaunchRegs = 96;
// Each type's share of the passes and of the other warps, as measured: no share makes any instance spill, but the compiler orders the passes
// otherwise under each.  us of a backward, 112 and 32 / 104 and 64 / 96 everywhere: bfloat16 64 pairs of 4096 positions 2012 / 2019 / 2045,
// 8 of 3000 210.8 / 210.9 / 214.3; float16 2064 / 2025 / 2074, 216.8 / 209.8 / 218.2, 15 of 777 72.4 / 70.5 / 72.6.
template <typename T> struct SplitRegs { static constexpr int passes = 112, others = 32; };
template <> struct SplitRegs<__half> { static constexpr int passes = 104, others = 64; };
template <typename T> constexpr bool split_regs_fit() { return kSplitWorkers * SplitRegs<T>::passes + 128 * SplitRegs<T>::others <= kSplitThreads * kSplitLaunchRegs; }
static_assert(split_regs_fit<__half>() && split_regs_fit<__nv_bfloat16>(), "setmaxnreg would wait forever");

// Events: named barriers on which the passes' `threads` arrive and go on, and one warp besides waits.  Such a barrier counts arrivals,
// whoever makes them, and sees no abort flag: a warp that arrived again before its last arrival there was taken would upset the count and
// leave the waiting warp in it for ever.  In ordinary flow an mbarrier wait lies between the two, for a product that is issued after the
// first was taken.  A wait that ends without its phase (the abort flag) shows nothing of the kind.  So the warp then stops working
// and makes the arrivals that are left, in their order, as full participants (ev_wait): each holds it until the event is taken, and with it
// all before.  What remains is that the first of these must not lie on a barrier where an arrival of this warp's may still be untaken; the
// events of a step take turns on a few barriers for that, which also keeps the ordinary flow's arrivals apart.  Every warp
// still makes every arrival once and in the same order, and the taking warps' other waits end by the flag, so all of them come through.
// (mbarriers of one arrival a warp instead, and bounded waits for them: the dim_head-64 kernel at B=4 N=4096 H=16 1931 -> 2127 us,
// 1024 pairs of one block 112 -> 131, dim_head 128 at B=2 H=8 N=1333 91.6 -> 98.  The taking warps publish how far they are
// and the others wait for that: 1940 -> 2005, a store before or after each bar.sync of the issuing warp.)
__device__ __forceinline__ void ev_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads + 32) : "memory"); }
__device__ __forceinline__ void ev_wait(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads + 32) : "memory"); }
// The arrival when a thread's accumulator columns are in registers.  Returns 0, read from shared memory behind it: the compiler
// moves an arrival behind arithmetic that does not depend on it, and the next product then starts a pass late, so a constant of
// the pass has this added to it (dim_head 64, B=4 N=4096 H=16: 2120 -> 1960 us; dim_head 128, 8 pairs of 8190: 1770 -> 1635).
__device__ __forceinline__ float ev_arrive_read(int id, int threads, const float* zero_s) {
  tc_fence_before();
  ev_arrive(id, threads);
  float zero;
  asm volatile("ld.volatile.shared.f32 %0, [%1];" : "=f"(zero) : "r"(smem_u32(zero_s)) : "memory");
  return zero;
}
// 0 if `kernel` was compiled to start with the registers that the sharing above counts on; asked once per kernel (`known`)
template <typename Kernel>
int check_launch_regs(Kernel kernel, std::atomic<bool>& known) {
  if (known.load(std::memory_order_relaxed)) return 0;
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kernel);
  if (e != cudaSuccess) return cuda_fail(e, "castle_bwd attribute");
  if (a.numRegs != kSplitLaunchRegs) return reject("castle_bwd: compiled with %d registers a thread instead of %d", a.numRegs, kSplitLaunchRegs);
  known.store(true, std::memory_order_relaxed);
  return 0;
}

// delta[b,h,i] = sum_d out * dout  (lookahead_keys_attention_triton.py:175-214 in the reference); clears the first NACC of the
// fp32 accumulators on the way (a memset of its own is a launch more).
template <typename T, int D, int NACC>
__global__ void castle_bwd_delta_kernel(const BwdParams p) {
  constexpr int LPR = D / 8;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / LPR) + threadIdx.x / LPR;
  const int sub = threadIdx.x % LPR;
  const int64_t total = (int64_t)p.B * p.H * p.N;
  float s = 0.f;
  if (row < total) {
    int bh = row / p.N, i = row % p.N, b = bh / p.H, h = bh % p.H;
    const T* po = reinterpret_cast<const T*>(p.out.ptr) + b * p.out.stride_b + h * p.out.stride_h + (int64_t)i * p.out.stride_n + sub * 8;
    const T* pd = reinterpret_cast<const T*>(p.dout.ptr) + b * p.dout.stride_b + h * p.dout.stride_h + (int64_t)i * p.dout.stride_n + sub * 8;
    uint4 a = *reinterpret_cast<const uint4*>(po), c = *reinterpret_cast<const uint4*>(pd);
    const uint32_t* ua = &a.x; const uint32_t* uc = &c.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 x = Elem<T>::unpack2(ua[j]), y = Elem<T>::unpack2(uc[j]);
      s += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (row < total && sub == 0) p.delta[row] = s;
  if (row < total) {
    float* const accs[3] = {p.acc_dqc, p.acc_dvu, p.acc_dku};
#pragma unroll
    for (int t = 0; t < NACC; ++t) {
      float4* a = reinterpret_cast<float4*>(accs[t] + row * D + sub * 8);
      a[0] = a[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// fp32 accumulators -> scaled 16-bit gradients in the caller's (strided) tensors.
// NACC = 3: dqc, dvu, dku (dqu is written by the kernel that owns the key block).
template <typename T, int D, int NACC>
__global__ void castle_bwd_finish_kernel(const BwdParams p) {
  constexpr int LPR = D / 8;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x / LPR) + threadIdx.x / LPR;
  const int sub = threadIdx.x % LPR;
  overlap_wait();   // launched while the sums are being written
  if (row >= (int64_t)p.B * p.H * p.N) return;
  int bh = row / p.N, i = row % p.N, b = bh / p.H, h = bh % p.H;
  const float* srcs[3] = {p.acc_dqc, p.acc_dvu, p.acc_dku};
  const castle_tensor_t* dsts[3] = {&p.dqc, &p.dvu, &p.dku};
#pragma unroll
  for (int t = 0; t < NACC; ++t) {
    const float4* s4 = reinterpret_cast<const float4*>(srcs[t] + row * D + sub * 8);
    float4 x = s4[0], y = s4[1];
    uint4 q;
    q.x = Elem<T>::pack2(x.x * p.scale, x.y * p.scale); q.y = Elem<T>::pack2(x.z * p.scale, x.w * p.scale);
    q.z = Elem<T>::pack2(y.x * p.scale, y.y * p.scale); q.w = Elem<T>::pack2(y.z * p.scale, y.w * p.scale);
    T* d = reinterpret_cast<T*>(dsts[t]->ptr) + b * dsts[t]->stride_b + h * dsts[t]->stride_h + (int64_t)i * dsts[t]->stride_n + sub * 8;
    *reinterpret_cast<uint4*>(d) = q;
  }
}

// dim_head 128 backward (bwd128.cu)
size_t bwd128_pair_bytes(int nblk);           // tile hand-over scratch of one (batch, head) pair
int bwd128_chunk_pairs(int BH, int nblk);     // pairs per launch pair that keep the scratch under its limit
int launch_bwd128(const BwdParams& p, int dtype, const CUtensorMap* in_maps, cudaStream_t st);

}  // namespace castle
