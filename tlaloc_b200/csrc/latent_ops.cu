// The row operations of a latent-attention layer: the pair of RMS norms in front of parallel mixer and feed-forward
// branches, the norms / rotation / cache write between the down- and up-projections, and interleaved RoPE.  Everything
// is evaluated in f32; only results are narrowed.
#include "common.cuh"

namespace tlaloc_b200 {
namespace {

// Sum over the CTA (blockDim.x a multiple of 32, at most 256); every thread gets it.
__device__ __forceinline__ float CtaSum(float v, float* red)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
  for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) r += red[w];
  return r;
}

__device__ __forceinline__ float InvRms(float sum_sq, int n, float eps)
{
  return 1.f / sqrtf(sum_sq / static_cast<float>(n) + eps);
}

__device__ __forceinline__ void Store4(float* o, float a, float b, float c, float d) { *reinterpret_cast<float4*>(o) = make_float4(a, b, c, d); }
__device__ __forceinline__ void Store4(__nv_bfloat16* o, float a, float b, float c, float d)
{
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  uint2 u;
  u.x = *reinterpret_cast<const uint32_t*>(&lo);
  u.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(o) = u;
}

// One CTA per row.  NI > 0: rows of up to 1024 NI values, a multiple of 4, 16-byte aligned: read once, kept in registers, NI words a thread and no more
// (the loads in flight bound it: registers that a row does not need are warps that an SM does not hold).
template <typename OT, int NI>
__global__ void __launch_bounds__(256) RmsNormPairKernel(const float* x, const float* gain_a, OT* out_a, const float* gain_b,
                                                         OT* out_b, int n, float eps)
{
  PrefetchL2(gain_a, n);
  PrefetchL2(gain_b, n);
  GridDependencySync();
  __shared__ float red[8];
  const size_t row = static_cast<size_t>(blockIdx.x) * n;
  const float* xr = x + row;
  if constexpr (NI > 0) {
    const int n4 = n >> 2;
    float4 v[NI];
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int j = threadIdx.x + i * 256;
      v[i] = j < n4 ? reinterpret_cast<const float4*>(xr)[j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NI; ++i) ss = fmaf(v[i].x, v[i].x, fmaf(v[i].y, v[i].y, fmaf(v[i].z, v[i].z, fmaf(v[i].w, v[i].w, ss))));
    const float inv = InvRms(CtaSum(ss, red), n, eps);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int j = threadIdx.x + i * 256;
      if (j >= n4) break;
      const float a = v[i].x * inv, b = v[i].y * inv, c = v[i].z * inv, d = v[i].w * inv;
      const float4 g = reinterpret_cast<const float4*>(gain_a)[j];
      Store4(out_a + row + 4 * j, a * g.x, b * g.y, c * g.z, d * g.w);
      if (out_b != nullptr) {
        const float4 h = reinterpret_cast<const float4*>(gain_b)[j];
        Store4(out_b + row + 4 * j, a * h.x, b * h.y, c * h.z, d * h.w);
      }
    }
  } else {
    float ss = 0.f;
    for (int j = threadIdx.x; j < n; j += 256) ss = fmaf(xr[j], xr[j], ss);
    const float inv = InvRms(CtaSum(ss, red), n, eps);
    for (int j = threadIdx.x; j < n; j += 256) {
      const float v = xr[j] * inv;
      out_a[row + j] = FromF32<OT>(v * gain_a[j]);
      if (out_b != nullptr) out_b[row + j] = FromF32<OT>(v * gain_b[j]);
    }
  }
}

// The pair (u, v) at an angle whose cosine and sine (with the design's magnitude already in them) are c and s.
__device__ __forceinline__ float2 Rotate(float u, float v, float c, float s)
{
  return make_float2(u * c - v * s, v * c + u * s);
}

// One CTA per token: two norms, one rotation, one cache row.  VEC: q_rank up to 2048, kv_rank up to 1024, both and rot_dim multiples of 4, and everything
// aligned: the row is read once, by 16-byte words.  2048 tokens of 1536 + 576 values: 11.1 us element by element (bound by their instructions), 6.4 so.
// Element by element the registers are bound, so that an SM holds eight CTAs: 2048 tokens of 2052 + 72 values 12.4 us with six, 10.5 with eight (700 tokens 5.7, 6.3).
template <typename T, bool VEC>
__global__ void __launch_bounds__(256, VEC ? 4 : 8) LatentKvWriteKernel(const float* in, int64_t ld, const float* q_gain, const float* kv_gain, float eps,
                                                           const int* positions, const float* cos_t, const float* sin_t, const int* slots,
                                                           T* cq, T* pool, int64_t pool_ld, int q_rank, int kv_rank, int rot_dim,
                                                           int rot_dims, int num_slots, int max_pos)
{
  PrefetchL2(q_gain, q_rank);
  PrefetchL2(kv_gain, kv_rank);
  GridDependencySync();
  __shared__ float red[8], red2[8];
  const int t = blockIdx.x, tid = threadIdx.x;
  const float* row = in + static_cast<size_t>(t) * ld;
  const float* kv = row + q_rank;
  const int slot = __ldg(slots + t), pos = min(max(__ldg(positions + t), 0), max_pos - 1), pairs = rot_dims >> 1;
  T* out = pool + static_cast<size_t>(slot) * pool_ld;
  const float* rot = kv + kv_rank;
  const bool there = slot >= 0 && slot < num_slots;
  if constexpr (VEC) {
    const int q4 = q_rank >> 2, k4 = kv_rank >> 2, r4 = rot_dim >> 2;
    auto word = [](const float* p, int j) { return reinterpret_cast<const float4*>(p)[j]; };
    auto square = [](float4 v) { return fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w))); };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 a0 = tid < q4 ? word(row, tid) : zero, a1 = tid + 256 < q4 ? word(row, tid + 256) : zero, k0 = tid < k4 ? word(kv, tid) : zero;
    // the last threads turn the rotated part: they have the least of the rest to do
    const int i = 255 - tid;
    float4 r = zero, cs = make_float4(1.f, 1.f, 1.f, 1.f), sn = zero;
    if (i < r4) {
      r = word(rot, i);
      if (4 * i < rot_dims) {  // one or two pairs
        const float *c = cos_t + static_cast<size_t>(pos) * pairs + 2 * i, *n = sin_t + static_cast<size_t>(pos) * pairs + 2 * i;
        cs.x = c[0], sn.x = n[0];
        if (4 * i + 2 < rot_dims) cs.y = c[1], sn.y = n[1];
      }
    }
    // both sums in one meeting of the warps
    float sq = square(a0) + square(a1), sk = square(k0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sq += __shfl_xor_sync(0xffffffffu, sq, o);
      sk += __shfl_xor_sync(0xffffffffu, sk, o);
    }
    if ((tid & 31) == 0) {
      red[tid >> 5] = sq;
      red2[tid >> 5] = sk;
    }
    __syncthreads();
    sq = sk = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      sq += red[w];
      sk += red2[w];
    }
    auto scaled = [&](T* o, int j, float4 v, float inv, const float* gain) {
      const float4 g = word(gain, j);
      Store4(o + 4 * j, v.x * inv * g.x, v.y * inv * g.y, v.z * inv * g.z, v.w * inv * g.w);
    };
    if (q_rank > 0) {
      const float inv = InvRms(sq, q_rank, eps);
      if (tid < q4) scaled(cq + static_cast<size_t>(t) * q_rank, tid, a0, inv, q_gain);
      if (tid + 256 < q4) scaled(cq + static_cast<size_t>(t) * q_rank, tid + 256, a1, inv, q_gain);
    }
    if (!there) return;
    if (tid < k4) scaled(out, tid, k0, InvRms(sk, kv_rank, eps), kv_gain);
    if (i < r4) {
      const float2 u = 4 * i < rot_dims ? Rotate(r.x, r.y, cs.x, sn.x) : make_float2(r.x, r.y);
      const float2 v = 4 * i + 2 < rot_dims ? Rotate(r.z, r.w, cs.y, sn.y) : make_float2(r.z, r.w);
      Store4(out + kv_rank + 4 * i, u.x, u.y, v.x, v.y);
    }
    return;
  }
  float sq = 0.f, sk = 0.f;
  for (int j = tid; j < q_rank; j += 256) sq = fmaf(row[j], row[j], sq);
  for (int j = tid; j < kv_rank; j += 256) sk = fmaf(kv[j], kv[j], sk);
  sq = CtaSum(sq, red);
  sk = CtaSum(sk, red2);
  if (q_rank > 0) {
    const float inv = InvRms(sq, q_rank, eps);
    for (int j = tid; j < q_rank; j += 256) cq[static_cast<size_t>(t) * q_rank + j] = FromF32<T>(row[j] * inv * q_gain[j]);
  }
  if (!there) return;
  const float inv = InvRms(sk, kv_rank, eps);
  for (int j = tid; j < kv_rank; j += 256) out[j] = FromF32<T>(kv[j] * inv * kv_gain[j]);
  for (int i = tid; i < pairs; i += 256) {
    const float2 r = Rotate(rot[2 * i], rot[2 * i + 1], cos_t[static_cast<size_t>(pos) * pairs + i], sin_t[static_cast<size_t>(pos) * pairs + i]);
    out[kv_rank + 2 * i] = FromF32<T>(r.x);
    out[kv_rank + 2 * i + 1] = FromF32<T>(r.y);
  }
  for (int j = rot_dims + tid; j < rot_dim; j += 256) out[kv_rank + j] = FromF32<T>(rot[j]);
}

__device__ __forceinline__ void LoadFour(const float* p, float* v)
{
  const float4 u = *reinterpret_cast<const float4*>(p);
  v[0] = u.x, v[1] = u.y, v[2] = u.z, v[3] = u.w;
}
__device__ __forceinline__ void LoadFour(const __nv_bfloat16* p, float* v)
{
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(u.x << 16), v[1] = __uint_as_float(u.x & 0xffff0000u), v[2] = __uint_as_float(u.y << 16), v[3] = __uint_as_float(u.y & 0xffff0000u);
}

// Two pairs a thread, where width and rot_dims are multiples of 4 and the rows start at whole fours: 2048 tokens of 32 heads of 64 11.2 us a pair
// at a time (bound by its instructions), 5.9 so.
template <typename T>
__global__ void __launch_bounds__(256) RopeInterleavedVecKernel(const T* in, int64_t in_t, int64_t in_h, T* out, int64_t out_t, int64_t out_h,
                                                                const int* positions, const float* cos_t, const float* sin_t, unsigned total,
                                                                unsigned heads, unsigned fours, int rot_dims, int max_pos)
{
  GridDependencySync();
  const unsigned i = blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const unsigned th = i / fours, f = i - th * fours, t = th / heads, h = th - t * heads;
  float v[4];
  LoadFour(in + t * in_t + h * in_h + 4 * f, v);
  if (static_cast<int>(4 * f) < rot_dims) {
    const int pos = min(max(__ldg(positions + t), 0), max_pos - 1);
    const size_t at = static_cast<size_t>(pos) * (rot_dims >> 1) + 2 * f;
    const float2 c = *reinterpret_cast<const float2*>(cos_t + at), s = *reinterpret_cast<const float2*>(sin_t + at);
    const float2 a = Rotate(v[0], v[1], c.x, s.x), b = Rotate(v[2], v[3], c.y, s.y);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  }
  Store4(out + t * out_t + h * out_h + 4 * f, v[0], v[1], v[2], v[3]);
}

// A thread per pair (or, past rot_dims, per two copied elements).
template <typename T>
__global__ void __launch_bounds__(256) RopeInterleavedKernel(const T* in, int64_t in_t, int64_t in_h, T* out, int64_t out_t, int64_t out_h,
                                                             const int* positions, const float* cos_t, const float* sin_t, long long total,
                                                             int heads, int width, int rot_dims, int max_pos)
{
  GridDependencySync();
  const long long i = static_cast<long long>(blockIdx.x) * 256 + threadIdx.x;
  if (i >= total) return;
  const int half = (width + 1) >> 1, pairs = rot_dims >> 1;
  const int p = static_cast<int>(i % half);
  const long long th = i / half;
  const int h = static_cast<int>(th % heads);
  const long long t = th / heads;
  const T* src = in + t * in_t + h * in_h + 2 * p;
  T* dst = out + t * out_t + h * out_h + 2 * p;
  if (p < pairs) {
    const int pos = min(max(__ldg(positions + t), 0), max_pos - 1);
    const float2 r = Rotate(ToF32(src[0]), ToF32(src[1]), cos_t[static_cast<size_t>(pos) * pairs + p], sin_t[static_cast<size_t>(pos) * pairs + p]);
    dst[0] = FromF32<T>(r.x);
    dst[1] = FromF32<T>(r.y);
  } else {
    dst[0] = src[0];
    if (2 * p + 1 < width) dst[1] = src[1];
  }
}

}  // namespace
}  // namespace tlaloc_b200

using namespace tlaloc_b200;

extern "C" int tlaloc_b200_rmsnorm_pair(const float* x, const float* gain_a, void* out_a, const float* gain_b, void* out_b,
                                        int32_t out_dtype, int32_t rows, int32_t n, float eps, void* stream)
{
  const char* op = "RMSNORM_PAIR";
  if (!x || !gain_a || !out_a || (out_b && !gain_b)) return Fail(kInvalid, "%s: a required device pointer is null", op);
  if (!IsFloatType(out_dtype)) return Fail(kInvalid, "%s: out must be f32 or bf16", op);
  if (rows < 0 || n < 1) return Fail(kInvalid, "%s: bad sizes", op);
  if (rows == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = n % 4 == 0 && n <= 8192 && Aligned16(x) && Aligned16(gain_a) && Aligned16(gain_b) && Aligned16(out_a) && Aligned16(out_b);
  cudaError_t e;
#define TLALOC_LAUNCH(OT, NI) \
  e = LaunchChained(RmsNormPairKernel<OT, NI>, rows, 256, 0, st, x, gain_a, static_cast<OT*>(out_a), gain_b, static_cast<OT*>(out_b), n, eps)
#define TLALOC_LAUNCH_NI(OT)                     \
  if (!vec) TLALOC_LAUNCH(OT, 0);                \
  else if (n <= 2 * 1024) TLALOC_LAUNCH(OT, 2);  \
  else if (n <= 3 * 1024) TLALOC_LAUNCH(OT, 3);  \
  else if (n <= 4 * 1024) TLALOC_LAUNCH(OT, 4);  \
  else TLALOC_LAUNCH(OT, 8)
  if (out_dtype == TLALOC_B200_F32) {
    TLALOC_LAUNCH_NI(float);
  } else {
    TLALOC_LAUNCH_NI(__nv_bfloat16);
  }
#undef TLALOC_LAUNCH_NI
#undef TLALOC_LAUNCH
  if (e != cudaSuccess) return CudaFail("RMSNORM_PAIR launch", e);
  CountLaunches(1);
  return kOk;
}

extern "C" int tlaloc_b200_latent_kv_write(const float* in, int64_t ld, const float* q_gain, const float* kv_gain, float eps,
                                           const int32_t* positions, const float* cos_table, const float* sin_table,
                                           const int32_t* slot_mapping, void* cq, void* pool, int32_t dtype, int64_t pool_ld,
                                           int32_t num_tokens, int32_t q_rank, int32_t kv_rank, int32_t rot_dim, int32_t rot_dims,
                                           int32_t num_slots, int32_t max_pos, void* stream)
{
  const char* op = "LATENT_KV_WRITE";
  if (!in || !kv_gain || !positions || !cos_table || !sin_table || !slot_mapping || !pool || (q_rank > 0 && (!q_gain || !cq))) {
    return Fail(kInvalid, "%s: a required device pointer is null", op);
  }
  if (!IsFloatType(dtype)) return Fail(kInvalid, "%s: the pool must be f32 or bf16", op);
  if (num_tokens < 0 || q_rank < 0 || kv_rank < 1 || rot_dim < 0 || num_slots < 1 || max_pos < 1) return Fail(kInvalid, "%s: bad sizes", op);
  if (rot_dims < 0 || rot_dims % 2 != 0 || rot_dims > rot_dim) {
    return Fail(kInvalid, "%s: %d rotated dimensions; an even number up to %d", op, rot_dims, rot_dim);
  }
  if (ld < static_cast<int64_t>(q_rank) + kv_rank + rot_dim || pool_ld < static_cast<int64_t>(kv_rank) + rot_dim) {
    return Fail(kInvalid, "%s: a row stride is shorter than its row", op);
  }
  if (num_tokens == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool vec = q_rank <= 2048 && kv_rank <= 1024 && rot_dim <= 1024 && q_rank % 4 == 0 && kv_rank % 4 == 0 && rot_dim % 4 == 0 && ld % 4 == 0 &&
                   pool_ld % 4 == 0 && Aligned16(in) && Aligned16(pool) && Aligned16(kv_gain) && (q_rank == 0 || (Aligned16(cq) && Aligned16(q_gain)));
  cudaError_t e;
#define TLALOC_LAUNCH(T, VEC)                                                                                                         \
  e = LaunchChained(LatentKvWriteKernel<T, VEC>, num_tokens, 256, 0, st, in, ld, q_gain, kv_gain, eps, positions, cos_table, sin_table, \
                    slot_mapping, static_cast<T*>(cq), static_cast<T*>(pool), pool_ld, q_rank, kv_rank, rot_dim, rot_dims, num_slots, max_pos)
  if (dtype == TLALOC_B200_F32) {
    if (vec) TLALOC_LAUNCH(float, true);
    else TLALOC_LAUNCH(float, false);
  } else {
    if (vec) TLALOC_LAUNCH(__nv_bfloat16, true);
    else TLALOC_LAUNCH(__nv_bfloat16, false);
  }
#undef TLALOC_LAUNCH
  if (e != cudaSuccess) return CudaFail("LATENT_KV_WRITE launch", e);
  CountLaunches(1);
  return kOk;
}

extern "C" int tlaloc_b200_rope_interleaved(const void* in, int64_t in_ld_token, int64_t in_ld_head, void* out, int64_t out_ld_token,
                                            int64_t out_ld_head, int32_t dtype, const int32_t* positions, const float* cos_table,
                                            const float* sin_table, int32_t num_tokens, int32_t num_heads, int32_t width,
                                            int32_t rot_dims, int32_t max_pos, void* stream)
{
  const char* op = "ROPE_INTERLEAVED";
  if (!in || !out || !positions || !cos_table || !sin_table) return Fail(kInvalid, "%s: a required device pointer is null", op);
  if (!IsFloatType(dtype)) return Fail(kInvalid, "%s: f32 or bf16", op);
  if (num_tokens < 0 || num_heads < 1 || width < 1 || max_pos < 1) return Fail(kInvalid, "%s: bad sizes", op);
  if (rot_dims < 0 || rot_dims % 2 != 0 || rot_dims > width) return Fail(kInvalid, "%s: %d rotated dimensions; an even number up to %d", op, rot_dims, width);
  if (num_tokens == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const uintptr_t four = 4 * DtypeBytes(dtype);
  if (width % 4 == 0 && rot_dims % 4 == 0 && in_ld_token % 4 == 0 && in_ld_head % 4 == 0 && out_ld_token % 4 == 0 && out_ld_head % 4 == 0 &&
      reinterpret_cast<uintptr_t>(in) % four == 0 && reinterpret_cast<uintptr_t>(out) % four == 0 && reinterpret_cast<uintptr_t>(cos_table) % 8 == 0 &&
      reinterpret_cast<uintptr_t>(sin_table) % 8 == 0 && static_cast<long long>(num_tokens) * num_heads * (width / 4) < (1ll << 31)) {
    const unsigned all = static_cast<unsigned>(num_tokens) * num_heads * (width / 4);
#define TLALOC_LAUNCH(T)                                                                                                                                 \
  LaunchChained(RopeInterleavedVecKernel<T>, (all + 255) / 256, 256, 0, st, static_cast<const T*>(in), in_ld_token, in_ld_head, static_cast<T*>(out),    \
                out_ld_token, out_ld_head, positions, cos_table, sin_table, all, static_cast<unsigned>(num_heads), static_cast<unsigned>(width / 4), rot_dims, max_pos)
    const cudaError_t e = dtype == TLALOC_B200_F32 ? TLALOC_LAUNCH(float) : TLALOC_LAUNCH(__nv_bfloat16);
#undef TLALOC_LAUNCH
    if (e != cudaSuccess) return CudaFail("ROPE_INTERLEAVED launch", e);
    CountLaunches(1);
    return kOk;
  }
  const long long total = static_cast<long long>(num_tokens) * num_heads * ((width + 1) / 2);
  const unsigned blocks = static_cast<unsigned>((total + 255) / 256);
  cudaError_t e;
#define TLALOC_LAUNCH(T)                                                                                                           \
  e = LaunchChained(RopeInterleavedKernel<T>, blocks, 256, 0, st, static_cast<const T*>(in), in_ld_token, in_ld_head,              \
                    static_cast<T*>(out), out_ld_token, out_ld_head, positions, cos_table, sin_table, total, num_heads, width, rot_dims, max_pos)
  if (dtype == TLALOC_B200_F32) TLALOC_LAUNCH(float);
  else TLALOC_LAUNCH(__nv_bfloat16);
#undef TLALOC_LAUNCH
  if (e != cudaSuccess) return CudaFail("ROPE_INTERLEAVED launch", e);
  CountLaunches(1);
  return kOk;
}
