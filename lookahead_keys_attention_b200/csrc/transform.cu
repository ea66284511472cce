// Element-wise passes around the parallel kernels, for callers whose tensors the kernels do not take (or do not
// give back) as they are: another element type (fp16 operands for fp32 callers and for bf16 callers at long
// sequences), another row width (zero-padded heads), rotary embedding, or decode caches the forward kernels
// cannot fill from their operand tiles.  ONE pass does all of it for up to six tensors: for each row
//     y = round_src(rotate(x)) * mul,   dst = convert(y),   copy = round_src(rotate(x))
// so that a rotary layer costs one launch instead of about eighty element-wise torch launches, and a long prompt
// one instead of a conversion and four cache copies.  HBM-bound: 8 elements (16 or 32 bytes) per thread and access.
#include <type_traits>

#include "common.cuh"
#include "rotary.cuh"
#include "vec.cuh"

namespace castle {

struct TransformParams {
  castle_tensor_t src[6], dst[6], copy[6];   // ptr of dst / copy may be null
  int count, H, N;
  int src_d, dst_d, cpr;                     // row widths; cpr = 16-byte-of-8-elements chunks per row = max(width) / 8
  int rows;                                  // positions per block
  uint32_t per_row_inv, heads_inv;           // see quotient()
  uint32_t rot_mask;                         // which of the tensors are rotated
  RotaryParams rot;
  const float* mul;
};

constexpr int kTransformThreads = 256, kTransformLines = 4;
constexpr int kTransformTable = 2048;   // cos/sin pairs a block keeps in shared memory

// x / d by a multiplication with inv = ceil(2^32 / d), exact for x * d < 2^32; inv = 0: a plain division (d of 1, or beyond 2^15)
__host__ inline uint32_t inverse_of(int d) { return d > 1 && d <= 1 << 15 ? (uint32_t)((((uint64_t)1 << 32) + d - 1) / d) : 0; }
__device__ __forceinline__ int quotient(int x, int d, uint32_t inv) { return inv ? (int)__umulhi((uint32_t)x, inv) : x / d; }

// One block: `rows` consecutive positions of one batch entry, all heads and tensors of them, so that a position's
// cosines and sines are computed once and used count * H times.
template <typename S, typename D, bool ROT>
__global__ void __launch_bounds__(kTransformThreads, 4) castle_transform_kernel(const TransformParams p) {
  __shared__ float2 table[ROT ? kTransformTable : 1];
  const int nblocks = (p.N + p.rows - 1) / p.rows;
  const int b = blockIdx.x / nblocks, n0 = (blockIdx.x % nblocks) * p.rows;
  const int nrows = min(p.rows, p.N - n0);
  const int half = (ROT ? (p.src_d < p.dst_d ? p.src_d : p.dst_d) : 2) / 2;   // pairs of the rotated width
  if constexpr (ROT) {
    for (int i = threadIdx.x; i < nrows * half; i += kTransformThreads)
      table[i] = rotary_cos_sin(p.rot, n0 + i / half, rotary_freq(p.rot, i % half));
    __syncthreads();
  }
  const float mul = p.mul ? *p.mul : 1.f;
  // A line is one tensor's row of one head; p.cpr adjacent threads take it, a thread kTransformLines of them at a time: their
  // loads are on their way together, as they lie, and no index needs a division.  Six tensors, one access at a time with four
  // divisions / so: 1 x 16 x 8190 x 128 bf16 to fp16 93 / 75 us (5.4 TB/s), 1 x 32 x 16384 x 128 335 / 280, 2 x 8 x 8192 x 32 padded to
  // 64 45 / 34, 4 x 16 x 4096 x 64 rotated 131 / 118, 2 x 8 x 4096 x 64 fp32 to fp16 31 / 28.  (Held as floats instead of as they
  // lie, the four cost so many registers that the first took 131.)
  const int per_row = p.count * p.H, lines = nrows * per_row, step = kTransformThreads / p.cpr;
  const int c8 = (int)(threadIdx.x % p.cpr) * 8, first = threadIdx.x / p.cpr;
  if (first >= step) return;
  for (int l0 = first; l0 < lines; l0 += step * kTransformLines) {
    Raw8<S> raw[kTransformLines];
#pragma unroll
    for (int u = 0; u < kTransformLines; ++u) {
      const int l = l0 + u * step, r = quotient(l, per_row, p.per_row_inv), th = l - r * per_row, t = quotient(th, p.H, p.heads_inv), h = th - t * p.H;
      if (l < lines && c8 < p.src_d) {
        const castle_tensor_t& s = p.src[t];
        raw[u] = *reinterpret_cast<const Raw8<S>*>(reinterpret_cast<const S*>(s.ptr) + b * s.stride_b + h * s.stride_h + (int64_t)(n0 + r) * s.stride_n + c8);
      } else {
        raw[u] = Raw8<S>{};   // zeros
      }
    }
#pragma unroll
    for (int u = 0; u < kTransformLines; ++u) {
      const int l = l0 + u * step;
      if (l >= lines) break;
      float v[8];
      load8<S>(reinterpret_cast<const S*>(&raw[u]), v);
      const int r = quotient(l, per_row, p.per_row_inv), th = l - r * per_row, t = quotient(th, p.H, p.heads_inv), h = th - t * p.H, n = n0 + r;
      if (ROT && (p.rot_mask >> t & 1) && c8 < p.src_d && c8 < 2 * half) {
        if (p.rot.inverse) rotate8<float>(v, table + r * half + c8 / 2);   // a gradient: no rounding before the factor
        else rotate8<S>(v, table + r * half + c8 / 2);
      }
      const castle_tensor_t& k = p.copy[t];
      if (k.ptr && c8 < p.src_d)
        store8<S>(reinterpret_cast<S*>(k.ptr) + b * k.stride_b + h * k.stride_h + (int64_t)n * k.stride_n + c8, v);
      const castle_tensor_t& d = p.dst[t];
      if (d.ptr && c8 < p.dst_d) {
        if (p.mul) {
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] *= mul;
        }
        // Saturate instead of overflowing.  With a factor the values are an upstream gradient's, which castle_amax_scale has
        // brought into range: an infinity there is the caller's own and stays one, as loss scalers look for it.
        if (std::is_same<D, __half>::value && !std::is_same<S, __half>::value) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            v[j] = v[j] != v[j] || (p.mul && fabsf(v[j]) == INFINITY) ? v[j] : fminf(fmaxf(v[j], -65504.f), 65504.f);
        }
        store8<D>(reinterpret_cast<D*>(d.ptr) + b * d.stride_b + h * d.stride_h + (int64_t)n * d.stride_n + c8, v);
      }
    }
  }
}

// The largest finite |x| of a tensor and from it the power of two that brings a gradient to a fixed magnitude:
// out[0] = s = 2^e, the largest power of two <= 64 / max (e at most 24, so that zeros stay harmless), out[1] = 1 / s.
// Infinities and NaN have no part in it: one of them leaves the other rows' gradients as they are without it.  `state` is
// two zeroed words (running maximum as bits of a non-negative float, blocks done) that the last block zeroes again.
template <typename S>
__global__ void __launch_bounds__(256) castle_amax_scale_kernel(const S* __restrict__ x, int64_t n8, uint32_t* state, float* out) {
  float m = 0.f;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n8; i += (int64_t)gridDim.x * 256) {
    float v[8];
    load8<S>(x + i * 8, v);
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fabsf(v[j]) < INFINITY ? fmaxf(m, fabsf(v[j])) : m;
  }
  uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
  __shared__ uint32_t warp_bits[8];
  if ((threadIdx.x & 31) == 0) warp_bits[threadIdx.x >> 5] = bits;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) bits = max(bits, warp_bits[w]);
    atomicMax(state, bits);
    __threadfence();
    if (atomicAdd(state + 1, 1u) == gridDim.x - 1) {
      const float amax = fmaxf(__uint_as_float(atomicExch(state, 0u)), 1e-30f);
      state[1] = 0u;
      int e;
      frexpf(64.f / amax, &e);
      e = min(e - 1, 24);
      out[0] = ldexpf(1.f, e);
      out[1] = ldexpf(1.f, -e);
    }
  }
}

template <typename S, typename D>
static void launch_transform(const TransformParams& p, int B, cudaStream_t st) {
  const unsigned grid = (unsigned)B * ((p.N + p.rows - 1) / p.rows);
  if (p.rot.freqs) castle_transform_kernel<S, D, true><<<grid, kTransformThreads, 0, st>>>(p);
  else castle_transform_kernel<S, D, false><<<grid, kTransformThreads, 0, st>>>(p);
}
template <typename S>
static void launch_transform_s(const TransformParams& p, int B, int dst_dtype, cudaStream_t st) {
  if (dst_dtype == CASTLE_BF16) launch_transform<S, __nv_bfloat16>(p, B, st);
  else if (dst_dtype == CASTLE_F16) launch_transform<S, __half>(p, B, st);
  else launch_transform<S, float>(p, B, st);
}

}  // namespace castle

using namespace castle;

extern "C" int castle_transform(const castle_problem_t* p, int32_t count, const castle_tensor_t* src,
                                const castle_tensor_t* dst, int32_t dst_dtype, int32_t dst_dim_head,
                                const castle_tensor_t* copies, const castle_rotary_t* rotary, uint32_t rotary_mask,
                                const float* mul, void* stream) {
  const char* who = "castle_transform";
  if (!p || !src || !dst) return reject("%s: null argument", who);
  if (p->batch <= 0 || p->heads <= 0 || p->seq_len <= 0) return reject("%s: empty problem", who);
  if (count < 1 || count > 6) return reject("%s: %d tensors (1 to 6)", who, count);
  if (p->dtype < CASTLE_BF16 || p->dtype > CASTLE_F32 || dst_dtype < CASTLE_BF16 || dst_dtype > CASTLE_F32)
    return reject("%s: unknown dtype", who);
  const int sd = p->dim_head, dd = dst_dim_head;
  if (sd < 8 || dd < 8 || sd > 128 || dd > 128 || sd % 8 || dd % 8)
    return reject("%s: dim_head %d -> %d not supported (multiples of 8 up to 128)", who, sd, dd);
  int rc = 0;
  TransformParams t;
  t.count = count; t.H = p->heads; t.N = p->seq_len; t.src_d = sd; t.dst_d = dd; t.cpr = (sd > dd ? sd : dd) / 8;
  for (int i = 0; i < 6; ++i) {
    const castle_tensor_t none{nullptr, 0, 0, 0};
    t.src[i] = i < count ? src[i] : none;
    t.dst[i] = i < count ? dst[i] : none;
    t.copy[i] = i < count && copies ? copies[i] : none;
    if (i >= count) continue;
    if (!tensor_ok(&t.src[i], p->dtype, "source", &rc)) return rc;
    if (t.dst[i].ptr && !tensor_ok(&t.dst[i], dst_dtype, "destination", &rc)) return rc;
    if (t.copy[i].ptr && !tensor_ok(&t.copy[i], p->dtype, "copy", &rc)) return rc;
  }
  t.rot = RotaryParams{nullptr, CASTLE_F32, 0, 0.f};
  t.rot_mask = 0;
  if (rotary && rotary->freqs) {
    if (rotary->dtype < CASTLE_BF16 || rotary->dtype > CASTLE_F32) return reject("%s: unknown rotary dtype", who);
    t.rot = RotaryParams{rotary->freqs, rotary->dtype, rotary->inverse, (float)rotary->position0};
    t.rot_mask = rotary_mask;
  }
  t.mul = mul;
  t.per_row_inv = inverse_of(count * p->heads);
  t.heads_inv = inverse_of(p->heads);
  // positions per block: about twelve accesses per thread where that leaves eight blocks per SM, within the cosine table
  const int64_t positions = (int64_t)p->batch * p->seq_len;
  t.rows = 3072 / (count * p->heads * t.cpr);
  if (t.rows > positions / (148 * 8)) t.rows = (int)(positions / (148 * 8));
  if (t.rows > kTransformTable / 64) t.rows = kTransformTable / 64;
  if (t.rows < 1) t.rows = 1;
  if ((int64_t)p->batch * ((p->seq_len + t.rows - 1) / t.rows) > 2147483647LL) return reject("%s: grid too large", who);
  cudaStream_t st = (cudaStream_t)stream;
  if (p->dtype == CASTLE_BF16) launch_transform_s<__nv_bfloat16>(t, p->batch, dst_dtype, st);
  else if (p->dtype == CASTLE_F16) launch_transform_s<__half>(t, p->batch, dst_dtype, st);
  else launch_transform_s<float>(t, p->batch, dst_dtype, st);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_transform launch");
}

extern "C" int castle_amax_scale(int32_t dtype, const void* x, int64_t count, uint32_t* state, float* out, void* stream) {
  if (dtype < CASTLE_BF16 || dtype > CASTLE_F32) return reject("castle_amax_scale: unknown dtype");
  if (!x || !state || !out || count <= 0) return reject("castle_amax_scale: null pointer or empty tensor");
  if (count % 8 || ((uintptr_t)x) % 16) return reject("castle_amax_scale: count must be a multiple of 8 and x 16-byte aligned");
  const int64_t n8 = count / 8, want = (n8 + 1023) / 1024;   // four accesses per thread, at most four blocks per SM
  const unsigned blocks = (unsigned)(want < 148 * 4 ? want : 148 * 4);
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == CASTLE_BF16) castle_amax_scale_kernel<<<blocks, 256, 0, st>>>((const __nv_bfloat16*)x, n8, state, out);
  else if (dtype == CASTLE_F16) castle_amax_scale_kernel<<<blocks, 256, 0, st>>>((const __half*)x, n8, state, out);
  else castle_amax_scale_kernel<<<blocks, 256, 0, st>>>((const float*)x, n8, state, out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : cuda_fail(e, "castle_amax_scale launch");
}
