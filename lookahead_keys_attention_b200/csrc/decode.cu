// Cached single-token CASTLE step (HBM-bound).
//
// Per (batch, head) the step streams four caches of `t` rows once: it reads
// qu_cache, U, kc_cache and vc_cache and writes U back, i.e. 5*t*d elements,
// which is the algorithmic traffic of the step.  Each row is handled by d/VEC
// adjacent lanes (VEC = 16 bytes of elements per lane), so every global access
// is a 128-bit load/store and a warp touches whole 128-byte lines; the three
// dot products of a row are reduced with xor-shuffles inside that lane group.
// Rows are split over `nsplit` CTAs per (batch, head); each CTA keeps a running
// (max, sum, weighted value sum) and writes one partial, which a small second
// kernel merges.
#include <algorithm>
#include <mutex>
#include "common.cuh"
#include "decode_row.cuh"

namespace castle {

struct DecodeParams {
  castle_tensor_t qc, kc, vc, qu, ku, vu;          // new rows
  castle_tensor_t U, quc, kcc, vcc;                // caches
  castle_tensor_t out;
  float* part;                                     // [BH][nsplit][2 + D]
  int H, t, nsplit, rows_per_split;
  float scale;
  int32_t* status;
  RotaryParams rot;                                // rotation of the new rows (all but vc); freqs null = none
  bool overlap;                                    // launched before the kernel that writes the new rows has ended
  uint32_t* counters;                              // [BH] zeroed: CTAs of a pair that are done; null = merge kernel
};

#ifndef CASTLE_DECODE_THREADS
#define CASTLE_DECODE_THREADS 128
#endif
#ifndef CASTLE_DECODE_UNROLL
#define CASTLE_DECODE_UNROLL 1
#endif
#ifndef CASTLE_DECODE_MIN_CTAS
#define CASTLE_DECODE_MIN_CTAS 8
#endif
constexpr int kDecodeThreads = CASTLE_DECODE_THREADS;
constexpr int kDecodeUnroll = CASTLE_DECODE_UNROLL;
constexpr int kMaxSplits = 64;   // CTAs that share the rows of one (batch, head) pair
static_assert(kDecodeThreads == 128, "decode_merge maps 128 threads to the columns of a head");

template <typename T, int D>
__device__ __forceinline__ void decode_store_out(const DecodeParams& p, int bh, int c, float v) {
  T* o = reinterpret_cast<T*>(p.out.ptr) + (bh / p.H) * p.out.stride_b + (bh % p.H) * p.out.stride_h;
  if constexpr (sizeof(T) == 4) o[c] = v;
  else o[c] = Elem<T>::from_f(v);
}

// Merge the partials of one (batch, head) pair, by a whole CTA of kDecodeThreads: the weights of the parts once
// per CTA into shared memory, then D columns x (threads / D) groups of parts, eight loads of a thread in flight.
template <typename T, int D>
__device__ __forceinline__ void decode_merge(const DecodeParams& p, int bh) {
  constexpr int G = kDecodeThreads / D;
  __shared__ float s_w[kMaxSplits], s_sum[G][D];
  const int nsplit = p.nsplit;
  const float* src = p.part + (int64_t)bh * nsplit * (2 + D);
  const int lane = threadIdx.x & 31;
  // every warp finds the maximum and the sum over the (at most 64) parts by itself
  const float m0 = lane < nsplit ? __ldcg(src + lane * (2 + D)) : -INFINITY;
  const float m1 = lane + 32 < nsplit ? __ldcg(src + (lane + 32) * (2 + D)) : -INFINITY;
  const float l0 = lane < nsplit ? __ldcg(src + lane * (2 + D) + 1) : 0.f;
  const float l1 = lane + 32 < nsplit ? __ldcg(src + (lane + 32) * (2 + D) + 1) : 0.f;
  float mm = fmaxf(m0, m1);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
  const float w0 = m0 == -INFINITY ? 0.f : __expf(m0 - mm), w1 = m1 == -INFINITY ? 0.f : __expf(m1 - mm);
  float ll = l0 * w0 + l1 * w1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
  if (threadIdx.x < 32) { s_w[lane] = w0; s_w[lane + 32] = w1; }
  __syncthreads();
  const int c = threadIdx.x % D, g = threadIdx.x / D;
  float a = 0.f;
#pragma unroll 8
  for (int s = g; s < nsplit; s += G) a += __ldcg(src + s * (2 + D) + 2 + c) * s_w[s];
  if constexpr (G > 1) {
    s_sum[g][c] = a;
    __syncthreads();
    if (g == 0) {
#pragma unroll
      for (int k = 1; k < G; ++k) a += s_sum[k][c];
    }
  }
  if (g == 0) decode_store_out<T, D>(p, bh, c, a / ll);
}

// End of both step kernels: merge the lane groups of a warp, then the warps of the CTA.  A pair whose rows were split
// leaves a partial; the CTA that leaves a pair's last one (p.counters) merges them, which saves the merge kernel's
// launch and its wait for the whole grid (3 to 8 us a step).
template <typename T, int D>
__device__ __forceinline__ void decode_finish(const DecodeParams& p, int bh, int split, float m, float l, float* acc) {
  constexpr int VEC = Vec<T>::N, LPR = D / VEC, NW = kDecodeThreads / 32;
  __shared__ float s_m[NW], s_l[NW], s_acc[NW][D];
  __shared__ bool s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPR, grp = lane / LPR;
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
    const float mn = fmaxf(m, m2);
    const float c1 = (m == -INFINITY) ? 0.f : __expf(m - mn), c2 = (m2 == -INFINITY) ? 0.f : __expf(m2 - mn);
    l = l * c1 + l2 * c2;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const float a2 = __shfl_xor_sync(0xffffffffu, acc[i], o);
      acc[i] = acc[i] * c1 + a2 * c2;
    }
    m = mn;
  }
  if (grp == 0) {
    if (sub == 0) { s_m[warp] = m; s_l[warp] = l; }
#pragma unroll
    for (int i = 0; i < VEC; ++i) s_acc[warp][sub * VEC + i] = acc[i];
  }
  __syncthreads();
  if (threadIdx.x < D) {
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < NW; ++w) mm = fmaxf(mm, s_m[w]);
    float ll = 0.f, aa = 0.f;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const float c = (s_m[w] == -INFINITY) ? 0.f : __expf(s_m[w] - mm);
      ll += s_l[w] * c;
      aa += s_acc[w][threadIdx.x] * c;
    }
    if (p.nsplit == 1) {
      decode_store_out<T, D>(p, bh, threadIdx.x, aa / ll);
    } else {
      float* dst = p.part + ((int64_t)bh * p.nsplit + split) * (2 + D);
      if (threadIdx.x == 0) { dst[0] = mm; dst[1] = ll; }
      dst[2 + threadIdx.x] = aa;
    }
  }
  if (p.nsplit == 1 || p.counters == nullptr) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(p.counters + bh, 1u) == (uint32_t)p.nsplit - 1;
    if (s_last) p.counters[bh] = 0;   // ready for the next launch
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  decode_merge<T, D>(p, bh);
}

template <typename T, int D>
__global__ void __launch_bounds__(kDecodeThreads, CASTLE_DECODE_MIN_CTAS) castle_decode_kernel(const DecodeParams p) {
  constexpr int VEC = Vec<T>::N;
  constexpr int LPR = D / VEC;                 // lanes per row
  constexpr int RPW = 32 / LPR;                // rows per warp per pass
  constexpr int NW = kDecodeThreads / 32;
  const int bh = blockIdx.x, split = blockIdx.y;
  const int b = bh / p.H, h = bh % p.H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPR, grp = lane / LPR;
  const int64_t col = (int64_t)sub * VEC;

  auto row_ptr = [&](const castle_tensor_t& t, int64_t r) {
    return reinterpret_cast<T*>(t.ptr) + b * t.stride_b + h * t.stride_h + r * t.stride_n + col;
  };

  overlap_next();
  overlap_wait();   // the new rows may come from the launch before (the caches do not)
  float qcv[VEC], kuv[VEC], vuv[VEC];
  Vec<T>::load(row_ptr(p.qc, 0), qcv);
  Vec<T>::load(row_ptr(p.ku, 0), kuv);
  Vec<T>::load(row_ptr(p.vu, 0), vuv);
  rotate_new<T>(p.rot, col, qcv, kuv, vuv);
#pragma unroll
  for (int i = 0; i < VEC; ++i) { qcv[i] *= p.scale; kuv[i] *= p.scale; }  // scale*(qu.ku) == qu.(scale*ku)

  float m = -INFINITY, l = 0.f, acc[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[i] = 0.f;

  const int r_begin = split * p.rows_per_split;
  const int r_end = min(p.t, r_begin + p.rows_per_split);

  // rows of this CTA, RPW*NW*UNROLL per pass
  // (the loop bound is warp-uniform: the shuffles below need every lane of the warp)
  for (int base = r_begin + warp * RPW; base < r_end; base += RPW * NW * kDecodeUnroll) {
    float quv[kDecodeUnroll][VEC], uv[kDecodeUnroll][VEC], kv[kDecodeUnroll][VEC], vv[kDecodeUnroll][VEC];
    bool live[kDecodeUnroll];
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      int r = base + grp + u * RPW * NW;
      live[u] = r < r_end;
      if (live[u]) {
        Vec<T>::load(row_ptr(p.quc, r), quv[u]);
        Vec<T>::load(row_ptr(p.U, r), uv[u]);
        Vec<T>::load(row_ptr(p.kcc, r), kv[u]);
        Vec<T>::load(row_ptr(p.vcc, r), vv[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < kDecodeUnroll; ++u) {
      int r = base + grp + u * RPW * NW;
      float z = 0.f, sc = 0.f, su = 0.f;
      if (live[u]) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) z += quv[u][i] * kuv[i];
      }
      z = group_sum<LPR>(z);
      float a = sigmoid_f(z);
      if (live[u]) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) uv[u][i] += a * vuv[i];
        Vec<T>::round(uv[u]);
        Vec<T>::store(row_ptr(p.U, r), uv[u]);
#pragma unroll
        for (int i = 0; i < VEC; ++i) { sc += qcv[i] * kv[u][i]; su += qcv[i] * uv[u][i]; }
      }
      sc = group_sum<LPR>(sc);
      su = group_sum<LPR>(su);
      if (live[u]) {
        float s = sc - su * sigmoid_f(su);
        float mn = fmaxf(m, s);
        float corr = __expf(m - mn), pe = __expf(s - mn);
        l = l * corr + pe;
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] = acc[i] * corr + pe * vv[u][i];
        m = mn;
      }
    }
  }

  // the appended row: U[t] = 0 so its score is just qc.kc_new; done by the last split
  if (split == p.nsplit - 1 && warp == 0) {  // whole warp runs the shuffle; lane group 0 keeps the result
    float kn[VEC], vn[VEC], qn[VEC], zero[VEC];
    Vec<T>::load(row_ptr(p.kc, 0), kn);
    Vec<T>::load(row_ptr(p.vc, 0), vn);
    Vec<T>::load(row_ptr(p.qu, 0), qn);
    rotate_new<T>(p.rot, col, kn, qn, nullptr);
#pragma unroll
    for (int i = 0; i < VEC; ++i) zero[i] = 0.f;
    if (grp == 0) {
      Vec<T>::store(row_ptr(p.kcc, p.t), kn);
      Vec<T>::store(row_ptr(p.vcc, p.t), vn);
      Vec<T>::store(row_ptr(p.quc, p.t), qn);
      Vec<T>::store(row_ptr(p.U, p.t), zero);
    }
    float sc = 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) sc += qcv[i] * kn[i];
    sc = group_sum<LPR>(sc);
    if (grp == 0) {
      float mn = fmaxf(m, sc);
      float corr = __expf(m - mn), pe = __expf(sc - mn);
      l = l * corr + pe;
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[i] = acc[i] * corr + pe * vn[i];
      m = mn;
    }
  }

  decode_finish<T, D>(p, bh, split, m, l, acc);
}

// ---------------------------------------------------------------------------------------------
// Same step, with the four caches brought in by bulk asynchronous copies (the TMA engine) into a
// ring of shared-memory stages instead of per-thread loads: the bytes in flight no longer depend
// on how many warps are resident or on how many registers a thread can spare.  One thread issues,
// per stage, four contiguous copies (the rows of a tile are adjacent in each cache, which is why
// this variant needs position stride == dim_head); the warps consume a stage row group by row
// group, write U back from registers, and the stage is refilled after a block-wide barrier.
constexpr int kRingStages = 3;
// Rows per stage: 4 KB of each cache (fewer and larger copies for narrow heads), at least 16.
template <typename T, int D> struct RingRows { static constexpr int fit = 4096 / (D * (int)sizeof(T)), value = fit > 16 ? fit : 16; };

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <typename T, int D>
__global__ void __launch_bounds__(kDecodeThreads, 4) castle_decode_ring_kernel(const DecodeParams p) {
  constexpr int VEC = Vec<T>::N;
  constexpr int LPR = D / VEC;
  constexpr int RPW = 32 / LPR;
  constexpr int NW = kDecodeThreads / 32;
  constexpr int kRingRows = RingRows<T, D>::value;
  constexpr int PASSES = (kRingRows + RPW * NW - 1) / (RPW * NW);
  constexpr uint32_t ROWB = D * sizeof(T);
  constexpr uint32_t TENB = kRingRows * ROWB;            // one tensor's tile
  extern __shared__ __align__(128) uint8_t ring[];       // [stage][tensor: qu, U, kc, vc][row][D]
  __shared__ uint64_t full[kRingStages];
  __shared__ int abort_flag;

  const int bh = blockIdx.x, split = blockIdx.y;
  const int b = bh / p.H, h = bh % p.H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane % LPR, grp = lane / LPR;
  const int64_t col = (int64_t)sub * VEC;
  volatile int* abortp = &abort_flag;

  auto row_ptr = [&](const castle_tensor_t& t, int64_t r) {
    return reinterpret_cast<T*>(t.ptr) + b * t.stride_b + h * t.stride_h + r * t.stride_n + col;
  };
  const int r_begin = split * p.rows_per_split;
  const int r_end = min(p.t, r_begin + p.rows_per_split);
  const int ntiles = (max(r_end - r_begin, 0) + kRingRows - 1) / kRingRows;

  auto issue = [&](int tile) {  // thread 0 only
    const int st = tile % kRingStages;
    const int r0 = r_begin + tile * kRingRows;
    const uint32_t bytes = (uint32_t)min(kRingRows, r_end - r0) * ROWB;
    uint8_t* dst = ring + (size_t)st * 4 * TENB;
    mbar_expect_tx(&full[st], 4 * bytes);
    bulk_load(dst, row_ptr(p.quc, r0) - col, bytes, &full[st]);
    bulk_load(dst + TENB, row_ptr(p.U, r0) - col, bytes, &full[st]);
    bulk_load(dst + 2 * TENB, row_ptr(p.kcc, r0) - col, bytes, &full[st]);
    bulk_load(dst + 3 * TENB, row_ptr(p.vcc, r0) - col, bytes, &full[st]);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kRingStages; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
    abort_flag = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int t0 = 0; t0 < kRingStages && t0 < ntiles; ++t0) issue(t0);

  overlap_next();
  overlap_wait();   // the new rows may come from the launch before (the caches do not)
  float qcv[VEC], kuv[VEC], vuv[VEC];
  Vec<T>::load(row_ptr(p.qc, 0), qcv);
  Vec<T>::load(row_ptr(p.ku, 0), kuv);
  Vec<T>::load(row_ptr(p.vu, 0), vuv);
  rotate_new<T>(p.rot, col, qcv, kuv, vuv);
#pragma unroll
  for (int i = 0; i < VEC; ++i) { qcv[i] *= p.scale; kuv[i] *= p.scale; }

  float m = -INFINITY, l = 0.f, acc[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[i] = 0.f;

  for (int tile = 0; tile < ntiles; ++tile) {
    const int st = tile % kRingStages;
    mbar_wait(&full[st], (uint32_t)((tile / kRingStages) & 1), abortp);
    // A wait that ran out means this stage never arrived: the U cache is persistent state, so
    // nothing computed from such a stage may be stored.  (No early exit: the barrier below must
    // still be reached by every thread.)
    const bool arrived = (*abortp == 0);
    const uint8_t* src = ring + (size_t)st * 4 * TENB;
    const int r0 = r_begin + tile * kRingRows;
#pragma unroll
    for (int ps = 0; ps < PASSES; ++ps) {
      const int rr = ps * RPW * NW + warp * RPW + grp;   // row inside the tile
      const int r = r0 + rr;
      const bool live = arrived && rr < kRingRows && r < r_end;
      float quv[VEC], uv[VEC], kv[VEC], vv[VEC];
      if (live) {
        const T* base = reinterpret_cast<const T*>(src) + (size_t)rr * D + col;
        Vec<T>::load(base, quv);
        Vec<T>::load(base + kRingRows * D, uv);
        Vec<T>::load(base + 2 * kRingRows * D, kv);
        Vec<T>::load(base + 3 * kRingRows * D, vv);
      }
      float z = 0.f, sc = 0.f, su = 0.f;
      if (live) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) z += quv[i] * kuv[i];
      }
      z = group_sum<LPR>(z);
      const float a = sigmoid_f(z);
      if (live) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) uv[i] += a * vuv[i];
        Vec<T>::round(uv);
        Vec<T>::store(row_ptr(p.U, r), uv);
#pragma unroll
        for (int i = 0; i < VEC; ++i) { sc += qcv[i] * kv[i]; su += qcv[i] * uv[i]; }
      }
      sc = group_sum<LPR>(sc);
      su = group_sum<LPR>(su);
      if (live) {
        const float s = sc - su * sigmoid_f(su);
        const float mn = fmaxf(m, s);
        const float corr = __expf(m - mn), pe = __expf(s - mn);
        l = l * corr + pe;
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] = acc[i] * corr + pe * vv[i];
        m = mn;
      }
    }
    __syncthreads();  // every warp is done with this stage
    if (threadIdx.x == 0 && tile + kRingStages < ntiles) issue(tile + kRingStages);
  }

  // the appended row: U[t] = 0 so its score is just qc.kc_new; done by the last split
  if (split == p.nsplit - 1 && warp == 0) {
    float kn[VEC], vn[VEC], qn[VEC], zero[VEC];
    Vec<T>::load(row_ptr(p.kc, 0), kn);
    Vec<T>::load(row_ptr(p.vc, 0), vn);
    Vec<T>::load(row_ptr(p.qu, 0), qn);
    rotate_new<T>(p.rot, col, kn, qn, nullptr);
#pragma unroll
    for (int i = 0; i < VEC; ++i) zero[i] = 0.f;
    if (grp == 0 && *abortp == 0) {   // a timed-out step leaves the caches as they were
      Vec<T>::store(row_ptr(p.kcc, p.t), kn);
      Vec<T>::store(row_ptr(p.vcc, p.t), vn);
      Vec<T>::store(row_ptr(p.quc, p.t), qn);
      Vec<T>::store(row_ptr(p.U, p.t), zero);
    }
    float sc = 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) sc += qcv[i] * kn[i];
    sc = group_sum<LPR>(sc);
    if (grp == 0) {
      const float mn = fmaxf(m, sc);
      const float corr = __expf(m - mn), pe = __expf(sc - mn);
      l = l * corr + pe;
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[i] = acc[i] * corr + pe * vn[i];
      m = mn;
    }
  }

  decode_finish<T, D>(p, bh, split, m, l, acc);
  if (threadIdx.x == 0 && abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

template <typename T, int D>
__global__ void __launch_bounds__(kDecodeThreads) castle_decode_merge_kernel(const DecodeParams p) {
  overlap_wait();   // launched while the partials are being written (8 x 16 heads x 8191 positions: 229.2 -> 228.3 us a step)
  decode_merge<T, D>(p, blockIdx.x);
}

// How many CTAs share the rows of one (batch, head) pair.  The kernel is bandwidth bound and runs
// CASTLE_DECODE_MIN_CTAS CTAs per SM, so what matters is that the grid fills whole "waves" of
// resident CTAs: pick the smallest split (at least 128 rows each, at most 64) whose last wave is
// nearly full.
static int decode_nsplit(int BH, int t, int ctas_per_sm = CASTLE_DECODE_MIN_CTAS) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0)
      sms = n;
    else
      sms = 148;
  }
  const int slots = sms * ctas_per_sm;
  int max_ns = t / 128;
  if (max_ns > 64) max_ns = 64;
  if (max_ns < 1) max_ns = 1;
  int best = 1;
  double best_eff = 0.0;
  for (int ns = 1; ns <= max_ns; ++ns) {
    const long long total = (long long)BH * ns;
    const long long waves = (total + slots - 1) / slots;
    const double eff = (double)total / (double)(waves * slots);
    if (eff > best_eff + 0.02) { best_eff = eff; best = ns; }
  }
  return best;
}

constexpr int kRingCtasPerSm = 4;

// The ring kernel's split, bf16 us per step as the rule above has it / as this one does (pairs x positions x dim_head):
// 400 x 4000 x 64 205 / 174, 200 x 4000 x 64 109 / 97, 128 x 4000 x 64 71 / 65, 256 x 4000 x 64 128 / 116, 1024 x 8191 x 128
// 1654 / 1593, 700 x 8191 x 128 1148 / 1091, 64 x 8191 x 128 121 / 118; single runs of one size differ by 2 %.  A grid of one
// wave merges in the kernel and pays a CTA's start once, so it is taken where it fills its wave to 85 % and a CTA's share of
// the caches is at most 1 MB, or 2 MB where the wave is full: longer walks of a single wave drift apart (256 x 8191 x 128 431 us
// against 411, 592 x 1500 x 128 181 against 187).  Otherwise shares of at most 1 MB, as few as come within 5 % of the fullest
// last wave: chasing the last percent with finer shares cost more in starts than it gained.
static int decode_nsplit_ring(int BH, int t, int row_bytes) {
  const int64_t slots = 148 * kRingCtasPerSm, most = 1 << 20;
  const int one = (int)std::min<int64_t>(64, slots / BH);
  const int64_t filled = (int64_t)BH * one * 100;
  if (one >= 1 && t / one >= 128 && filled >= slots * 85 && (int64_t)t * row_bytes <= (filled >= slots * 97 ? 2 : 1) * most * one) return one;
  const int max_ns = std::max(1, std::min(64, t / 128));
  auto eff = [&](int ns) {
    const int64_t total = (int64_t)BH * ns, waves = (total + slots - 1) / slots;
    return (double)total / (double)(waves * slots);
  };
  const int least = (int)std::min<int64_t>(max_ns, ((int64_t)t * row_bytes + most - 1) / most);
  double best = 0.0;
  for (int ns = std::max(1, least); ns <= max_ns; ++ns) best = std::max(best, eff(ns));
  for (int ns = std::max(1, least); ns <= max_ns; ++ns)
    if (eff(ns) >= best - 0.05) return ns;
  return 1;
}

// The same for steps that leave SMs idle at 128 rows per CTA (few pairs, short caches): there a CTA's serial walk over
// its rows is the time, so the rows are cut as fine as two ring stages (32 rows) while the grid stays within one wave.
// row_bytes: a position's bytes in the four caches.
static int decode_nsplit_fine(int BH, int t, int ctas_per_sm, int row_bytes) {
  const int best = ctas_per_sm == kRingCtasPerSm ? decode_nsplit_ring(BH, t, row_bytes) : decode_nsplit(BH, t, ctas_per_sm);
  const int64_t slots = 148 * ctas_per_sm;
  if ((int64_t)BH * best >= slots) return best;
  int ns = (t + 31) / 32;
  if (ns > slots / BH) ns = (int)(slots / BH);
  if (ns > kMaxSplits) ns = kMaxSplits;
  return ns > best ? ns : best;
}

// The bulk-copy variant needs rows that are adjacent in memory.
static bool decode_use_ring(int D, const castle_tensor_t* const* caches) {
  for (int i = 0; i < 4; ++i)
    if (caches[i]->stride_n != D) return false;
  return true;
}

template <typename T, int D>
static int launch_decode(const DecodeParams& p, int BH, bool ring, cudaStream_t st) {
  dim3 grid(BH, p.nsplit);
  if (ring) {
    constexpr size_t smem = (size_t)kRingStages * 4 * RingRows<T, D>::value * D * sizeof(T);
    cudaError_t e = cudaFuncSetAttribute(castle_decode_ring_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "castle_decode_step attribute");
    ev_start(CASTLE_KERNEL_DECODE, st);
    e = launch_kernel(castle_decode_ring_kernel<T, D>, grid, kDecodeThreads, smem, st, p.overlap, p);
    if (e != cudaSuccess) return cuda_fail(e, "castle_decode_step launch");
    ev_stop(CASTLE_KERNEL_DECODE, st);
    if (p.nsplit > 1 && !p.counters) e = launch_kernel(castle_decode_merge_kernel<T, D>, dim3(BH), kDecodeThreads, 0, st, true, p);
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? 0 : cuda_fail(e, "castle_decode_step launch");
  }
  ev_start(CASTLE_KERNEL_DECODE, st);
  cudaError_t e = launch_kernel(castle_decode_kernel<T, D>, grid, kDecodeThreads, 0, st, p.overlap, p);
  if (e != cudaSuccess) return cuda_fail(e, "castle_decode_step launch");
  ev_stop(CASTLE_KERNEL_DECODE, st);
  if (p.nsplit > 1 && !p.counters) e = launch_kernel(castle_decode_merge_kernel<T, D>, dim3(BH), kDecodeThreads, 0, st, true, p);
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_decode_step launch");
}

template <typename T>
static int launch_decode_d(const DecodeParams& p, int BH, int D, bool ring, cudaStream_t st) {
  switch (D) {
    case 16: return launch_decode<T, 16>(p, BH, ring, st);
    case 32: return launch_decode<T, 32>(p, BH, ring, st);
    case 64: return launch_decode<T, 64>(p, BH, ring, st);
    case 128: return launch_decode<T, 128>(p, BH, ring, st);
  }
  return reject("castle_decode_step: dim_head %d not supported (16, 32, 64, 128)", D);
}

}  // namespace castle

using namespace castle;

// The (batch, head) pairs are the grid's first dimension.
static bool decode_pairs_ok(const castle_problem_t* p) {
  return p->batch > 0 && p->heads > 0 && (int64_t)p->batch * p->heads <= 2147483647LL;
}

extern "C" size_t castle_decode_workspace_bytes(const castle_problem_t* p, int32_t cache_len) {
  if (!p || !decode_pairs_ok(p)) return 0;
  int BH = p->batch * p->heads;
  const int row_bytes = 4 * p->dim_head * elem_size(p->dtype);
  int ns = decode_nsplit_fine(BH, cache_len, CASTLE_DECODE_MIN_CTAS, row_bytes), ns_ring = decode_nsplit_fine(BH, cache_len, kRingCtasPerSm, row_bytes);
  return (size_t)BH * (ns > ns_ring ? ns : ns_ring) * (2 + p->dim_head) * sizeof(float);
}

extern "C" int castle_decode_step(const castle_problem_t* p, int32_t cache_len, int32_t capacity,
                                  const castle_tensor_t* qc_new, const castle_tensor_t* kc_new,
                                  const castle_tensor_t* vc_new, const castle_tensor_t* qu_new,
                                  const castle_tensor_t* ku_new, const castle_tensor_t* vu_new,
                                  const castle_tensor_t* u_cache, const castle_tensor_t* qu_cache,
                                  const castle_tensor_t* kc_cache, const castle_tensor_t* vc_cache,
                                  const castle_tensor_t* out, void* workspace, size_t workspace_bytes,
                                  int32_t* status, void* stream) {
  return castle_decode_step_fused(p, cache_len, capacity, qc_new, kc_new, vc_new, qu_new, ku_new, vu_new, u_cache, qu_cache,
                                  kc_cache, vc_cache, out, nullptr, nullptr, 0, workspace, workspace_bytes, status, stream);
}

extern "C" int castle_decode_step_fused(const castle_problem_t* p, int32_t cache_len, int32_t capacity,
                                        const castle_tensor_t* qc_new, const castle_tensor_t* kc_new,
                                        const castle_tensor_t* vc_new, const castle_tensor_t* qu_new,
                                        const castle_tensor_t* ku_new, const castle_tensor_t* vu_new,
                                        const castle_tensor_t* u_cache, const castle_tensor_t* qu_cache,
                                        const castle_tensor_t* kc_cache, const castle_tensor_t* vc_cache,
                                        const castle_tensor_t* out, const castle_rotary_t* rotary, uint32_t* counters,
                                        int32_t overlap, void* workspace, size_t workspace_bytes, int32_t* status, void* stream) {
  if (!p) return reject("castle_decode_step: null problem");
  if (!decode_pairs_ok(p)) return reject("castle_decode_step: empty batch/heads, or more than 2^31 pairs");
  if (cache_len < 0 || cache_len >= capacity)
    return reject("castle_decode_step: cache_len %d must be in [0, capacity %d)", cache_len, capacity);
  if (p->dtype != CASTLE_BF16 && p->dtype != CASTLE_F16 && p->dtype != CASTLE_F32)
    return reject("castle_decode_step: unknown dtype %d", p->dtype);
  int rc = 0;
  const castle_tensor_t* ts[11] = {qc_new, kc_new, vc_new, qu_new, ku_new, vu_new, u_cache, qu_cache, kc_cache, vc_cache, out};
  const char* names[11] = {"qc_new", "kc_new", "vc_new", "qu_new", "ku_new", "vu_new", "u_cache", "qu_cache", "kc_cache", "vc_cache", "out"};
  for (int i = 0; i < 11; ++i)
    if (!tensor_ok(ts[i], p->dtype, names[i], &rc)) return rc;
  DecodeParams dp;
  dp.qc = *qc_new; dp.kc = *kc_new; dp.vc = *vc_new; dp.qu = *qu_new; dp.ku = *ku_new; dp.vu = *vu_new;
  dp.U = *u_cache; dp.quc = *qu_cache; dp.kcc = *kc_cache; dp.vcc = *vc_cache; dp.out = *out;
  int BH = p->batch * p->heads;
  dp.H = p->heads; dp.t = cache_len; dp.scale = p->scale; dp.status = status;
  const castle_tensor_t* caches[4] = {u_cache, qu_cache, kc_cache, vc_cache};
  const bool ring = status != nullptr && decode_use_ring(p->dim_head, caches);
  dp.nsplit = decode_nsplit_fine(BH, cache_len, ring ? kRingCtasPerSm : CASTLE_DECODE_MIN_CTAS, 4 * p->dim_head * elem_size(p->dtype));
  dp.rows_per_split = (cache_len + dp.nsplit - 1) / dp.nsplit;
  if (dp.rows_per_split < 1) dp.rows_per_split = 1;
  dp.part = (float*)workspace;
  // Merging in the step kernel costs every CTA a fence that waits for its U rows to land.  Within one wave of CTAs that
  // is hidden by the launch it saves (8 pairs x 771 rows: 12.5 us -> 11 us, and one launch less on the host); over several
  // waves it is not (128 pairs x 8191 rows, 8 waves: 231 us against 213 + 8 us with the merge kernel).
  const int64_t slots = 148 * (ring ? kRingCtasPerSm : CASTLE_DECODE_MIN_CTAS);
  dp.counters = (int64_t)BH * dp.nsplit <= slots ? counters : nullptr;
  dp.overlap = overlap != 0;
  dp.rot = RotaryParams{nullptr, CASTLE_F32, 0, 0.f};
  if (rotary && rotary->freqs) {
    if (rotary->dtype < CASTLE_BF16 || rotary->dtype > CASTLE_F32) return reject("castle_decode_step: unknown rotary dtype");
    dp.rot = RotaryParams{rotary->freqs, rotary->dtype, rotary->inverse, (float)rotary->position0};
  }
  if (dp.nsplit > 1) {
    size_t need = (size_t)BH * dp.nsplit * (2 + p->dim_head) * sizeof(float);
    if (!workspace || workspace_bytes < need)
      return reject("castle_decode_step: workspace too small (%zu < %zu bytes)", workspace_bytes, need);
  }
  cudaStream_t st = (cudaStream_t)stream;
  switch (p->dtype) {
    case CASTLE_BF16: return launch_decode_d<__nv_bfloat16>(dp, BH, p->dim_head, ring, st);
    case CASTLE_F16: return launch_decode_d<__half>(dp, BH, p->dim_head, ring, st);
    default: return launch_decode_d<float>(dp, BH, p->dim_head, ring, st);
  }
}

// ---------------------------------------------------------------------------
// Decode step for hosts that may not allocate device memory on the token path.
//
// Some callers of this library cannot hand over a scratch buffer: a serving
// loop whose own arena took all device memory at start-up (so a cudaMalloc on
// the token path would fail, and would stall the device even if it did not), or
// a small non-torch host that binds only this C ABI and has no device allocator
// of its own.  For them the split partials of the decode step live in a fixed
// array inside the library image.  Every GPU that loads the library carries
// this array (520 KiB) until the process exits.
namespace castle {

constexpr int kStaticMaxSlots = 1024;          // batch * heads * row-splits
constexpr int kStaticSlotFloats = 2 + 128;     // (max, sum) + dim_head values, dim_head <= 128
static __device__ __align__(256) float g_decode_static_scratch[kStaticMaxSlots * kStaticSlotFloats];

// In host code the array's name is only a handle for the runtime, not an address a kernel may
// use; the device address is looked up once per device and kept here.
constexpr int kMaxDevices = 64;
static float* g_decode_static_ptr[kMaxDevices] = {nullptr};
static std::mutex g_decode_static_mu;   // host threads may make their first call on a device at the same time

}  // namespace castle

extern "C" int castle_decode_step_static(const castle_problem_t* p, int32_t cache_len, int32_t capacity,
                                         const castle_tensor_t* qc_new, const castle_tensor_t* kc_new,
                                         const castle_tensor_t* vc_new, const castle_tensor_t* qu_new,
                                         const castle_tensor_t* ku_new, const castle_tensor_t* vu_new,
                                         const castle_tensor_t* u_cache, const castle_tensor_t* qu_cache,
                                         const castle_tensor_t* kc_cache, const castle_tensor_t* vc_cache,
                                         const castle_tensor_t* out, int32_t* status, void* stream) {
  if (!p) return reject("castle_decode_step_static: null problem");
  if (!decode_pairs_ok(p)) return reject("castle_decode_step_static: empty batch/heads, or more than 2^31 pairs");
  if (cache_len < 0 || cache_len >= capacity)
    return reject("castle_decode_step_static: cache_len %d must be in [0, capacity %d)", cache_len, capacity);
  if (p->dtype != CASTLE_BF16 && p->dtype != CASTLE_F16 && p->dtype != CASTLE_F32)
    return reject("castle_decode_step_static: unknown dtype %d", p->dtype);
  int rc = 0;
  const castle_tensor_t* ts[11] = {qc_new, kc_new, vc_new, qu_new, ku_new, vu_new, u_cache, qu_cache, kc_cache, vc_cache, out};
  const char* names[11] = {"qc_new", "kc_new", "vc_new", "qu_new", "ku_new", "vu_new", "u_cache", "qu_cache", "kc_cache", "vc_cache", "out"};
  for (int i = 0; i < 11; ++i)
    if (!tensor_ok(ts[i], p->dtype, names[i], &rc)) return rc;
  const int BH = p->batch * p->heads;
  const int nsplit = decode_nsplit(BH, cache_len);
  if (p->dim_head > 128 || (int64_t)BH * nsplit > kStaticMaxSlots)
    return reject("castle_decode_step_static: batch*heads*splits = %lld exceeds the built-in scratch of %d partials "
                  "(dim_head <= 128); use castle_decode_step with a caller-owned workspace",
                  (long long)BH * nsplit, kStaticMaxSlots);
  // set-up, once per device, with that device current
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "castle_decode_step_static cudaGetDevice");
  if (dev < 0 || dev >= kMaxDevices) return reject("castle_decode_step_static: device ordinal %d not supported", dev);
  float* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_decode_static_mu);
    if (g_decode_static_ptr[dev] == nullptr) {
      float* ptr = nullptr;
      e = cudaGetSymbolAddress((void**)&ptr, g_decode_static_scratch);
      if (e != cudaSuccess) return cuda_fail(e, "castle_decode_step_static cudaGetSymbolAddress");
      g_decode_static_ptr[dev] = ptr;
    }
    scratch = g_decode_static_ptr[dev];
  }
  DecodeParams dp;
  dp.qc = *qc_new; dp.kc = *kc_new; dp.vc = *vc_new; dp.qu = *qu_new; dp.ku = *ku_new; dp.vu = *vu_new;
  dp.U = *u_cache; dp.quc = *qu_cache; dp.kcc = *kc_cache; dp.vcc = *vc_cache; dp.out = *out;
  dp.H = p->heads; dp.t = cache_len; dp.scale = p->scale; dp.status = status;
  dp.nsplit = nsplit;
  dp.rows_per_split = (cache_len + nsplit - 1) / nsplit;
  if (dp.rows_per_split < 1) dp.rows_per_split = 1;
  // Every partial slot the merge kernel reads is written by this same call first, so the
  // array needs no clearing between calls even though it keeps the previous call's contents.
  dp.part = scratch;
  dp.counters = nullptr;
  dp.overlap = false;
  dp.rot = RotaryParams{nullptr, CASTLE_F32, 0, 0.f};
  cudaStream_t st = (cudaStream_t)stream;
  switch (p->dtype) {
    case CASTLE_BF16: return launch_decode_d<__nv_bfloat16>(dp, BH, p->dim_head, false, st);
    case CASTLE_F16: return launch_decode_d<__half>(dp, BH, p->dim_head, false, st);
    default: return launch_decode_d<float>(dp, BH, p->dim_head, false, st);
  }
}
