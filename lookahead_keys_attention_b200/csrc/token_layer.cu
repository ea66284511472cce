// A whole layer's cached single-token step as ONE launch, for the sizes where launches and the waits between them are the
// time: norm + projection, the step itself and the output projection were three launches (csrc/token_linear.cu,
// csrc/decode.cu), 13 us of GPU and 7 us of host time a token at 1 x 512, 8 heads, 771 positions, for 7 MB from L2.
//
// A cluster of eight CTAs owns one head of R batch rows and needs nothing from the other heads until the very end:
//   A  each CTA computes an eighth of the head's six new rows (its weight rows streamed with 16-byte loads, x normalised by
//      every CTA for itself) and writes them into the shared memory of all eight
//   B  8 / R CTAs share the cached rows of a batch row; bulk asynchronous copies bring them into shared memory, all of
//      them, while A runs.  The eight partial soft-max sums go to the shared memory of all eight again
//   C  each CTA merges them and computes an eighth of the outputs' share of this head.  The shares meet in global memory:
//      the last of the H CTAs that own the same outputs adds them up in the order of the heads
// The two hand-overs inside a cluster are hardware barriers of CTAs that are resident together; the one between heads
// waits for nobody, so heads that do not fit on the GPU at the same time cannot block each other.
//
// What bounds it is neither memory nor arithmetic: 16 k cycles at 1 x 512, 8 heads, 771 positions, bf16, are some ten
// dependent steps of 1.4 to 3.4 k (a trip to L2, a hand-over, a reduction), and code that runs once is fetched as it runs, some
// 16 cycles an instruction, which is why the merges spread over lanes instead of being unrolled and the new rows are rotated
// once per CTA (by every lane group for itself: 4 k cycles more).  us per token, three launches / one: this size 20.1 / 14.4
// called from Python and 14.7 / 10.0 replayed from a CUDA graph; 2 x 128 positions, fp32, 19.8 / 14.1 and 12.9 / 10.3;
// 15 heads x 128, 1000 positions, bf16, 24.8 / 18.9 and 22.2 / 18.9; 15 heads x 128, 300 positions, fp32, 69.7 / 30.8.
// A CTA handles 128 rows of 64 16-bit values in 2.4 k cycles, and at most 120 run: with caches that do not fit into their
// shared memory (castle_token_layer_fits) the three launches over the whole GPU are faster (8 heads, 16384 positions: 26.9
// against 34.3).
#include "common.cuh"
#include "decode_row.cuh"

namespace castle {

constexpr int kTlThreads = 512, kTlCluster = 8, kTlWarps = kTlThreads / 32;
constexpr int kTlClusters = 15;                               // so many run at the same time, with one CTA per SM
constexpr int kTlStages = 2, kTlRowsAtOnce = 2;               // rows that a lane group works on side by side
constexpr uint32_t kTlTensorBytes = kTlThreads * 16 * kTlRowsAtOnce;   // of a stage, per cache
constexpr uint32_t kTlRing = kTlStages * 4 * kTlTensorBytes;
constexpr int kTlMaxX = 8192;                                 // floats of x in shared memory

struct TokenLayerParams {
  const void *x, *norm, *wqkv, *wout;
  void* y;
  castle_tensor_t U, quc, kcc, vcc;
  float* part;          // [H][B][N]: a head's share of the outputs
  uint32_t* counters;   // [groups of R rows][8], zero before and after
  int B, H, K, N, t;    // N = outputs of the last projection
  int64_t ldx;
  float eps, scale;
  RotaryParams rot;
  int32_t* status;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// The same place in another CTA's shared memory
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

template <int D> __host__ __device__ constexpr int token_layer_slice(int N) { return (N + kTlCluster - 1) / kTlCluster; }
template <int D, int R> static size_t token_layer_smem(int K, int N) {
  const int xs = R * (K > token_layer_slice<D>(N) ? K : token_layer_slice<D>(N));
  return kTlRing + (size_t)(xs + R * 6 * D + kTlCluster * (D + 2) + R * D) * sizeof(float);
}

template <typename T, int D, int R>
__global__ void __cluster_dims__(kTlCluster, 1, 1) __launch_bounds__(kTlThreads, 1) castle_token_layer_kernel(const TokenLayerParams p) {
  constexpr int VEC = Vec<T>::N, LPR = D / VEC, RPW = 32 / LPR, U = kTlRowsAtOnce, PASS = RPW * kTlWarps, ROWS = U * PASS;   // lanes a row; rows of a warp, of the CTA, of a stage
  constexpr int NS = kTlCluster / R;                                                     // CTAs that share a batch row's cache
  constexpr int NEW = 6 * D, SHARE = NEW / kTlCluster, PER_WARP = (SHARE + kTlWarps - 1) / kTlWarps;   // weight rows of the head, a CTA, a warp
  constexpr uint32_t ROWB = D * sizeof(T);
  static_assert(ROWS * ROWB == kTlTensorBytes, "a stage is U passes");
  extern __shared__ __align__(128) uint8_t smem[];
  const int slice = token_layer_slice<D>(p.N), K = p.K;
  float* news = reinterpret_cast<float*>(smem + kTlRing);     // [R][6][D]: qu, ku, vu, qc, kc, vc, rounded to T
  float* parts = news + R * NEW;                              // [R][NS][D + 2]
  float* os = parts + kTlCluster * (D + 2);                   // [R][D]: the head's output, rounded to T
  float* xs = os + R * D;                                     // [R][K]; later the outputs' shares [R][slice]
  __shared__ uint64_t full[kTlStages];
  __shared__ int abort_flag;
  __shared__ float s_ss[kTlWarps][R], s_m[kTlWarps], s_l[kTlWarps], s_acc[kTlWarps][D];
  __shared__ float2 s_cs[D / 2];
  __shared__ bool s_last;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, sub = lane % LPR, grp = lane / LPR, col = sub * VEC;
  const int rank = blockIdx.x % kTlCluster, h = blockIdx.x / kTlCluster, b0 = blockIdx.y * R;
  const int r = rank % R, split = rank / R, b = b0 + r;
  const bool mine = b < p.B;
  const int per_split = (p.t + NS - 1) / NS, r_begin = split * per_split, r_end = mine ? min(p.t, r_begin + per_split) : r_begin;
  const int ntiles = (max(r_end - r_begin, 0) + ROWS - 1) / ROWS;
  volatile int* abortp = &abort_flag;
  auto row_ptr = [&](const castle_tensor_t& c, int row) {
    return reinterpret_cast<T*>(c.ptr) + b * c.stride_b + h * c.stride_h + (int64_t)row * D;
  };
  auto issue = [&](int st) {   // thread 0
    const int row = r_begin + st * ROWS;
    const uint32_t bytes = (uint32_t)min(ROWS, r_end - row) * ROWB;
    uint8_t* dst = smem + st * 4 * kTlTensorBytes;
    mbar_expect_tx(&full[st], 4 * bytes);
    bulk_g2s(dst, row_ptr(p.quc, row), bytes, &full[st]);
    bulk_g2s(dst + kTlTensorBytes, row_ptr(p.U, row), bytes, &full[st]);
    bulk_g2s(dst + 2 * kTlTensorBytes, row_ptr(p.kcc, row), bytes, &full[st]);
    bulk_g2s(dst + 3 * kTlTensorBytes, row_ptr(p.vcc, row), bytes, &full[st]);
  };
  if (tid == 0) {
    for (int s = 0; s < kTlStages; ++s) mbar_init(&full[s], 1);
    mbar_fence_init();
    abort_flag = 0;
  }
  __syncthreads();
  cluster_arrive();   // its shared memory may be written from now on
  overlap_next();
  overlap_wait();     // everything below reads what earlier launches may have written

  // ---- A: weight rows [rank * SHARE, ...) of the head's six new rows, PER_WARP per warp
  const int chunks = K / VEC;   // at most one per thread (castle_token_layer_fits)
  const int g0 = rank * SHARE + warp * PER_WARP, g_end = rank * SHARE + SHARE;
  const T* wbase = reinterpret_cast<const T*>(p.wqkv);
  auto w_ptr = [&](int g) { return reinterpret_cast<const uint4*>(wbase + ((int64_t)(g / D) * p.H * D + h * D + g % D) * K); };
  constexpr int PF = PER_WARP > 4 ? 2 : 4;   // chunks of each row in flight
  uint4 q[PF][PER_WARP];
  auto fetch = [&](int s, int c) {
    if (c < chunks) {
#pragma unroll
      for (int i = 0; i < PER_WARP; ++i) q[s][i] = w_ptr(min(g0 + i, g_end - 1))[c];
    }
  };
#pragma unroll
  for (int s = 0; s < PF; ++s) fetch(s, lane + 32 * s);
  const bool has_x = tid < chunks;
  uint4 xq[R], nq = make_uint4(0, 0, 0, 0);
  if (has_x) {
#pragma unroll
    for (int rr = 0; rr < R; ++rr)
      xq[rr] = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.x) + (int64_t)min(b0 + rr, p.B - 1) * p.ldx + tid * VEC);
    if (p.norm) nq = *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(p.norm) + tid * VEC);
  }
  if (tid == 0)
    for (int i = 0; i < ntiles; ++i) issue(i);
  if (p.rot.freqs && tid >= kTlThreads - D / 2) {   // (the last warps are not the ones that have issued the copies)
    const int i = tid - (kTlThreads - D / 2);
    s_cs[i] = rotary_cos_sin(p.rot, 0, rotary_freq(p.rot, i));
  }
  float total[R];
  if (p.norm) {
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      float ss = 0.f, v[VEC];
      if (has_x) {
        Vec<T>::unpack(xq[rr], v);
#pragma unroll
        for (int j = 0; j < VEC; ++j) ss = fmaf(v[j], v[j], ss);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (lane == 0) s_ss[warp][rr] = ss;
    }
    __syncthreads();
#pragma unroll
    for (int rr = 0; rr < R; ++rr) {
      float ss = s_ss[lane % kTlWarps][rr];
#pragma unroll
      for (int o = kTlWarps / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      total[rr] = ss;
    }
  }
#pragma unroll
  for (int rr = 0; rr < R; ++rr) {
    if (!has_x) break;
    float v[VEC];
    Vec<T>::unpack(xq[rr], v);
    if (p.norm) {
      float g[VEC];
      const float inv = rsqrtf(total[rr] / (float)K + p.eps);
      Vec<T>::unpack(nq, g);
#pragma unroll
      for (int j = 0; j < VEC; ++j) v[j] = round_to<T>(v[j] * inv * g[j]);   // the norm's result has the type of x
    }
#pragma unroll
    for (int j = 0; j < VEC; j += 4) *reinterpret_cast<float4*>(xs + rr * K + tid * VEC + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
  }
  __syncthreads();
  {
    float acc[PER_WARP][R];
#pragma unroll
    for (int i = 0; i < PER_WARP; ++i)
#pragma unroll
      for (int rr = 0; rr < R; ++rr) acc[i][rr] = 0.f;
    for (int c0 = 0; c0 < chunks; c0 += 32 * PF) {
#pragma unroll
      for (int s = 0; s < PF; ++s) {
        const int c = c0 + 32 * s + lane;
        if (c < chunks) {
          float wv[PER_WARP][VEC];
#pragma unroll
          for (int i = 0; i < PER_WARP; ++i) Vec<T>::unpack(q[s][i], wv[i]);
          fetch(s, c + 32 * PF);
#pragma unroll
          for (int rr = 0; rr < R; ++rr) {
#pragma unroll
            for (int j = 0; j < VEC; j += 4) {
              const float4 xv = *reinterpret_cast<const float4*>(xs + rr * K + c * VEC + j);
#pragma unroll
              for (int i = 0; i < PER_WARP; ++i) {
                acc[i][rr] = fmaf(wv[i][j], xv.x, acc[i][rr]);
                acc[i][rr] = fmaf(wv[i][j + 1], xv.y, acc[i][rr]);
                acc[i][rr] = fmaf(wv[i][j + 2], xv.z, acc[i][rr]);
                acc[i][rr] = fmaf(wv[i][j + 3], xv.w, acc[i][rr]);
              }
            }
          }
        }
      }
    }
    // the sums over the warp, then four values at a time to the eight CTAs
#pragma unroll
    for (int i = 0; i < PER_WARP; ++i)
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[i][rr] += __shfl_xor_sync(0xffffffffu, acc[i][rr], o);
      }
    cluster_wait();   // every CTA of the cluster runs
    const uint32_t dst = cluster_addr(news, lane & 7);
#pragma unroll
    for (int i = 0; i < PER_WARP; ++i)
#pragma unroll
      for (int rr = 0; rr < R; ++rr)
        if (((i * R + rr) & 3) == lane >> 3 && g0 + i < g_end) cluster_store(dst + (rr * NEW + g0 + i) * sizeof(float), round_to<T>(acc[i][rr]));
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  if (p.rot.freqs) {   // the batch row's new rows but vc, a pair per thread
    for (int i = tid; i < 5 * D / 2; i += kTlThreads) rotate_pair<T>(news[r * NEW + 2 * i], news[r * NEW + 2 * i + 1], s_cs[i % (D / 2)]);
    __syncthreads();
  }

  // ---- B: the step over this CTA's rows
  auto new_row = [&](int slot, float* v) {
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = news[r * NEW + slot * D + col + i];
  };
  float m = -INFINITY, l = 0.f, acc[VEC];
  {
    float qcv[VEC], kuv[VEC], vuv[VEC];
    new_row(3, qcv);
    new_row(1, kuv);
    new_row(2, vuv);
#pragma unroll
    for (int i = 0; i < VEC; ++i) { qcv[i] *= p.scale; kuv[i] *= p.scale; acc[i] = 0.f; }
    for (int st = 0; st < ntiles; ++st) {
      mbar_wait(&full[st], 0, abortp);
      // (what never arrived is not used and U not written from it; the barriers are still reached)
      const bool arrived = *abortp == 0;
      const int row0 = r_begin + st * ROWS + warp * RPW;   // + u * PASS + grp
      if (row0 < r_end) {                                    // the warp has rows (it shuffles as a whole)
        const bool both = row0 + PASS < r_end;
        float uv[U][VEC], sc[U], su[U], z[U];
        bool live[U];
        const T* base = reinterpret_cast<const T*>(smem + st * 4 * kTlTensorBytes) + (warp * RPW + grp) * D + col;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          live[u] = arrived && row0 + u * PASS + grp < r_end;
          z[u] = sc[u] = su[u] = 0.f;
          if (live[u]) {
            float v[VEC];
            Vec<T>::load(base + u * PASS * D, v);
            Vec<T>::load(base + (ROWS + u * PASS) * D, uv[u]);
#pragma unroll
            for (int i = 0; i < VEC; ++i) z[u] += v[i] * kuv[i];
            Vec<T>::load(base + (2 * ROWS + u * PASS) * D, v);
#pragma unroll
            for (int i = 0; i < VEC; ++i) sc[u] += qcv[i] * v[i];
          }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            z[u] += __shfl_xor_sync(0xffffffffu, z[u], o);
            sc[u] += __shfl_xor_sync(0xffffffffu, sc[u], o);
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const float a = sigmoid_f(z[u]);
          if (live[u]) {
#pragma unroll
            for (int i = 0; i < VEC; ++i) uv[u][i] += a * vuv[i];
            Vec<T>::round(uv[u]);
#pragma unroll
            for (int i = 0; i < VEC; ++i) su[u] += qcv[i] * uv[u][i];
            Vec<T>::store(row_ptr(p.U, row0 + u * PASS + grp) + col, uv[u]);
          }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
#pragma unroll
          for (int u = 0; u < U; ++u) su[u] += __shfl_xor_sync(0xffffffffu, su[u], o);
        }
        float s[U], mn = m;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          s[u] = live[u] ? sc[u] - su[u] * sigmoid_f(su[u]) : -INFINITY;
          mn = fmaxf(mn, s[u]);
        }
        if (live[0]) {   // (a lane group may have no row)
          const float corr = __expf(m - mn);
          l *= corr;
#pragma unroll
          for (int i = 0; i < VEC; ++i) acc[i] *= corr;
          m = mn;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (live[u] && (u == 0 || both)) {
              const float pe = __expf(s[u] - mn);
              float v[VEC];
              Vec<T>::load(base + (3 * ROWS + u * PASS) * D, v);
              l += pe;
#pragma unroll
              for (int i = 0; i < VEC; ++i) acc[i] += pe * v[i];
            }
          }
        }
      }
    }
    // the appended row: U[t] = 0, so its score is just qc.kc_new
    if (split == NS - 1 && warp == 0 && mine) {
      float kn[VEC], vn[VEC], qn[VEC], zero[VEC];
      new_row(4, kn);
      new_row(5, vn);
      new_row(0, qn);
#pragma unroll
      for (int i = 0; i < VEC; ++i) zero[i] = 0.f;
      if (grp == 0 && *abortp == 0) {   // a timed-out step leaves the caches as they were
        Vec<T>::store(row_ptr(p.kcc, p.t) + col, kn);
        Vec<T>::store(row_ptr(p.vcc, p.t) + col, vn);
        Vec<T>::store(row_ptr(p.quc, p.t) + col, qn);
        Vec<T>::store(row_ptr(p.U, p.t) + col, zero);
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
  }
  // merge the lane groups of a warp, then the warps; the CTA's sums go to all eight
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
    const float mn = fmaxf(m, m2);
    const float c1 = m == -INFINITY ? 0.f : __expf(m - mn), c2 = m2 == -INFINITY ? 0.f : __expf(m2 - mn);
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
    for (int i = 0; i < VEC; ++i) s_acc[warp][col + i] = acc[i];
  }
  __syncthreads();
  {
    constexpr int G = kTlThreads / D;   // threads of a column; each stores to every G-th CTA
    const int c = tid % D, g = tid / D;
    // every warp weighs the warps' sums for itself, a lane each
    const float mw = s_m[lane % kTlWarps];
    float mm = mw;
#pragma unroll
    for (int o = kTlWarps / 2; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
    const float ew = mw == -INFINITY ? 0.f : __expf(mw - mm);
    float ll = s_l[lane % kTlWarps] * ew, aa = 0.f;
#pragma unroll
    for (int o = kTlWarps / 2; o > 0; o >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, o);
#pragma unroll
    for (int w = 0; w < kTlWarps; ++w) aa += s_acc[w][c] * __shfl_sync(0xffffffffu, ew, w);
    float* dst = parts + (r * NS + split) * (D + 2);
    for (int k = g; k < kTlCluster; k += G) {
      cluster_store(cluster_addr(dst + 2 + c, k), aa);
      if (c == 0) { cluster_store(cluster_addr(dst, k), mm); cluster_store(cluster_addr(dst + 1, k), ll); }
    }
  }
  // the first output weights are fetched across the barrier
  constexpr int PW = 2;
  const int inner = p.H * D;
  const T* wo = reinterpret_cast<const T*>(p.wout) + h * D + col;
  auto out_row = [&](int jj) { return jj < slice && rank * slice + jj < p.N; };
  uint4 qw[PW];
#pragma unroll
  for (int s = 0; s < PW; ++s) {
    const int jj = s * PASS + warp * RPW + grp;
    if (out_row(jj)) qw[s] = *reinterpret_cast<const uint4*>(wo + (int64_t)(rank * slice + jj) * inner);
  }
  __syncwarp();
  cluster_arrive();
  cluster_wait();

  // ---- C: this head's share of outputs [rank * slice, ...)
  for (int e = tid; e < R * D; e += kTlThreads) {
    const float* src = parts + (e / D) * NS * (D + 2);
    float mm = -INFINITY, ll = 0.f, aa = 0.f;
#pragma unroll
    for (int s = 0; s < NS; ++s) mm = fmaxf(mm, src[s * (D + 2)]);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const float ms = src[s * (D + 2)], w = ms == -INFINITY ? 0.f : __expf(ms - mm);
      ll += src[s * (D + 2) + 1] * w;
      aa += src[s * (D + 2) + 2 + e % D] * w;
    }
    os[e] = round_to<T>(aa / ll);   // (rows past the batch: not used)
  }
  __syncthreads();
  for (int j0 = 0; j0 < slice; j0 += PW * PASS) {
#pragma unroll
    for (int s = 0; s < PW; ++s) {
      const int jj = j0 + s * PASS + warp * RPW + grp;
      float w[VEC], a[R];
      const bool live = out_row(jj);
      if (live) Vec<T>::unpack(qw[s], w);
      const int next = jj + PW * PASS;
      if (out_row(next)) qw[s] = *reinterpret_cast<const uint4*>(wo + (int64_t)(rank * slice + next) * inner);
#pragma unroll
      for (int rr = 0; rr < R; ++rr) {
        a[rr] = 0.f;
        if (live) {
#pragma unroll
          for (int i = 0; i < VEC; ++i) a[rr] = fmaf(w[i], os[rr * D + col + i], a[rr]);
        }
        a[rr] = group_sum<LPR>(a[rr]);
        if (live && sub == 0) xs[rr * slice + jj] = a[rr];
      }
    }
  }
  __syncthreads();
  const int j_begin = rank * slice, count = min(slice, p.N - j_begin);
  auto store_y = [&](int bb, int j, float v) {
    T* y = reinterpret_cast<T*>(p.y) + (int64_t)bb * p.N + j;
    if constexpr (sizeof(T) == 4) *y = v;
    else *y = Elem<T>::from_f(v);
  };
  const int rows = min(R, p.B - b0);
  if (p.H > 1) {
    for (int rr = 0; rr < rows; ++rr)
      for (int j = tid; j < count; j += kTlThreads) p.part[((int64_t)h * p.B + b0 + rr) * p.N + j_begin + j] = xs[rr * slice + j];
    __syncthreads();
    if (tid == 0) {   // releases the whole CTA's shares (the barrier orders them before), and acquires the other heads'
      uint32_t* counter = p.counters + blockIdx.y * kTlCluster + rank;
      uint32_t before;
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
      s_last = before == (uint32_t)p.H - 1;
      if (s_last) *counter = 0;   // ready for the next launch
    }
    __syncthreads();
    if (s_last) {
      for (int rr = 0; rr < rows; ++rr)
        for (int j = tid; j < count; j += kTlThreads) {
          const float* src = p.part + (int64_t)(b0 + rr) * p.N + j_begin + j;
          float a = 0.f;
#pragma unroll 8
          for (int k = 0; k < p.H; ++k) a += __ldcg(src + (int64_t)k * p.B * p.N);
          store_y(b0 + rr, j_begin + j, a);
        }
    }
  } else {
    for (int rr = 0; rr < rows; ++rr)
      for (int j = tid; j < count; j += kTlThreads) store_y(b0 + rr, j_begin + j, xs[rr * slice + j]);
  }
  if (tid == 0 && abort_flag) atomicOr(p.status, CASTLE_STATUS_WAIT_TIMEOUT);
}

template <typename T, int D, int R>
static int launch_token_layer(const TokenLayerParams& p, bool overlap, cudaStream_t st) {
  const size_t smem = token_layer_smem<D, R>(p.K, p.N);
  cudaError_t e = cudaFuncSetAttribute(castle_token_layer_kernel<T, D, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_fail(e, "castle_token_layer attribute");
  e = launch_kernel(castle_token_layer_kernel<T, D, R>, dim3(kTlCluster * p.H, (p.B + R - 1) / R), kTlThreads, smem, st, overlap, p);
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_token_layer launch");
}
template <typename T, int D>
static int launch_token_layer_r(const TokenLayerParams& p, int R, bool overlap, cudaStream_t st) {
  if constexpr (sizeof(T) == 4) {
    if (R == 4) return launch_token_layer<T, D, 4>(p, overlap, st);
  }
  return R == 1 ? launch_token_layer<T, D, 1>(p, overlap, st) : launch_token_layer<T, D, 2>(p, overlap, st);
}
template <typename T>
static int launch_token_layer_d(const TokenLayerParams& p, int D, int R, bool overlap, cudaStream_t st) {
  return D == 32 ? launch_token_layer_r<T, 32>(p, R, overlap, st) : D == 64 ? launch_token_layer_r<T, 64>(p, R, overlap, st)
                                                                            : launch_token_layer_r<T, 128>(p, R, overlap, st);
}

// Batch rows of a cluster: more of them read the weights less often, but share eight CTAs; as few as keep all clusters on
// the GPU at the same time (2 x 128 positions, 8 heads, fp32: 10.8 us with 8 clusters of two rows, 17.6 with 16 of one for
// 15 places).  Four rows only in fp32: 16-bit types have the tensor-core projections (csrc/token_linear.cu), whose three
// launches are faster there (4 x 500 positions, 8 heads, bf16: 13.1 us against 16.4; fp32, 250 positions: 17.1 against
// 16.9, 15 heads 25.4 against 24.4).  0: no number of rows fits.
static int token_layer_rows(int batch, int heads, int dtype) {
  for (int R = 1; R <= (dtype == CASTLE_F32 ? 4 : 2); R *= 2)
    if ((int64_t)heads * ((batch + R - 1) / R) <= kTlClusters) return R;
  return 0;
}

}  // namespace castle

using namespace castle;

extern "C" int castle_token_layer_fits(const castle_problem_t* p, int32_t cache_len, int32_t dim, int32_t out_features) {
  if (!p || p->dtype < CASTLE_BF16 || p->dtype > CASTLE_F32 || p->batch < 1 || p->heads < 1 || dim < 1 || dim % 8 || out_features < 1) return 0;
  if (p->dim_head != 32 && p->dim_head != 64 && p->dim_head != 128) return 0;
  const int R = token_layer_rows(p->batch, p->heads, p->dtype), es = elem_size(p->dtype);
  if (R == 0) return 0;
  const int64_t per_split = ((int64_t)cache_len * R + kTlCluster - 1) / kTlCluster, slice = ((int64_t)out_features + kTlCluster - 1) / kTlCluster;
  return per_split * p->dim_head * es <= (int64_t)kTlStages * kTlTensorBytes && (int64_t)dim * es <= kTlThreads * 16 && R * (int64_t)dim <= kTlMaxX &&
         R * slice <= kTlMaxX;
}

extern "C" size_t castle_token_layer_workspace_bytes(const castle_problem_t* p, int32_t out_features) {
  return p && p->batch > 0 && p->heads > 0 && out_features > 0 ? (size_t)p->heads * p->batch * out_features * sizeof(float) : 0;
}

extern "C" int castle_token_layer(const castle_problem_t* p, int32_t cache_len, int32_t capacity, int32_t dim, int32_t out_features,
                                  const void* x, int64_t row_stride, const void* norm_weight, float eps, const void* to_qkv,
                                  const void* combine, const castle_tensor_t* u_cache, const castle_tensor_t* qu_cache,
                                  const castle_tensor_t* kc_cache, const castle_tensor_t* vc_cache, const castle_rotary_t* rotary,
                                  void* y, uint32_t* counters, int32_t overlap, void* workspace, size_t workspace_bytes,
                                  int32_t* status, void* stream) {
  if (cache_len < 0 || cache_len >= capacity) return reject("castle_token_layer: cache_len %d must be in [0, capacity %d)", cache_len, capacity);
  if (!castle_token_layer_fits(p, cache_len, dim, out_features)) return reject("castle_token_layer: size not supported (see castle_token_layer_fits)");
  if (!x || !to_qkv || !combine || !y || !counters || !status) return reject("castle_token_layer: null tensor");
  const int es = elem_size(p->dtype);
  if (((uintptr_t)x | (uintptr_t)to_qkv | (uintptr_t)combine | (uintptr_t)norm_weight) % 16 || row_stride * es % 16)
    return reject("castle_token_layer: pointers and the row stride must be 16-byte aligned");
  int rc = 0;
  const castle_tensor_t* caches[4] = {u_cache, qu_cache, kc_cache, vc_cache};
  const char* names[4] = {"u_cache", "qu_cache", "kc_cache", "vc_cache"};
  for (int i = 0; i < 4; ++i) {
    if (!tensor_ok(caches[i], p->dtype, names[i], &rc)) return rc;
    if (caches[i]->stride_n != p->dim_head) return reject("%s: rows must be adjacent in memory", names[i]);
  }
  if (!workspace || workspace_bytes < castle_token_layer_workspace_bytes(p, out_features)) return reject("castle_token_layer: workspace too small");
  TokenLayerParams tp;
  tp.x = x; tp.norm = norm_weight; tp.wqkv = to_qkv; tp.wout = combine; tp.y = y;
  tp.U = *u_cache; tp.quc = *qu_cache; tp.kcc = *kc_cache; tp.vcc = *vc_cache;
  tp.part = (float*)workspace; tp.counters = counters;
  tp.B = p->batch; tp.H = p->heads; tp.K = dim; tp.N = out_features; tp.t = cache_len;
  tp.ldx = row_stride; tp.eps = eps; tp.scale = p->scale; tp.status = status;
  tp.rot = RotaryParams{nullptr, CASTLE_F32, 0, 0.f};
  if (rotary && rotary->freqs) {
    if (rotary->dtype < CASTLE_BF16 || rotary->dtype > CASTLE_F32) return reject("castle_token_layer: unknown rotary dtype");
    tp.rot = RotaryParams{rotary->freqs, rotary->dtype, rotary->inverse, (float)rotary->position0};
  }
  const int R = token_layer_rows(p->batch, p->heads, p->dtype);
  cudaStream_t st = (cudaStream_t)stream;
  if (p->dtype == CASTLE_BF16) return launch_token_layer_d<__nv_bfloat16>(tp, p->dim_head, R, overlap != 0, st);
  if (p->dtype == CASTLE_F16) return launch_token_layer_d<__half>(tp, p->dim_head, R, overlap != 0, st);
  return launch_token_layer_d<float>(tp, p->dim_head, R, overlap != 0, st);
}
