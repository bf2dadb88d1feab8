// Token ids into rows and rows into token ids (ir/.../inference/HfDecoderGraph.kt: embedding :904-909; greedy next token): what every
// model of the framework begins and ends a step with.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace tlaloc_b200 {
namespace {

namespace cg = cooperative_groups;
constexpr int kEmbedThreads = 128, kArgmaxThreads = 512, kArgmaxCluster = 8;

// A row of the table widened to f32, sixteen bytes of it per thread: blockIdx.y counts stretches of the row (as many as a grid has, then again).  A single CTA walking a row
// element by element was a chain of dim / 256 dependent trips (128 rows of 8192: 16.7 us; this form 3.8 us, 5.2 MB of traffic).
template <typename TT, bool VEC>
__global__ void __launch_bounds__(kEmbedThreads) EmbeddingKernel(const TT* table, const int* ids, float* out, int vocab, int dim)
{
  constexpr int kPer = 16 / static_cast<int>(sizeof(TT));
  GridDependencySync();
  const int p = blockIdx.x;
  int v = __ldg(ids + p);
  v = v < 0 ? 0 : (v >= vocab ? vocab - 1 : v);
  for (long long d0 = (static_cast<long long>(blockIdx.y) * kEmbedThreads + threadIdx.x) * kPer; d0 < dim; d0 += gridDim.y * kEmbedThreads * kPer) {
    const TT* src = table + static_cast<size_t>(v) * dim + d0;
    float* dst = out + static_cast<size_t>(p) * dim + d0;
    if (VEC) {
      const uint4 raw = __ldcg(reinterpret_cast<const uint4*>(src));  // L2: an f32 table may be rows that the kernel before has written
      const TT* e = reinterpret_cast<const TT*>(&raw);
#pragma unroll
      for (int i = 0; i < kPer; i += 4) {
        *reinterpret_cast<float4*>(dst + i) = make_float4(ToF32(e[i]), ToF32(e[i + 1]), ToF32(e[i + 2]), ToF32(e[i + 3]));
      }
    } else {
      for (int i = 0; i < kPer && d0 + i < dim; ++i) dst[i] = ToF32(src[i]);
    }
  }
}

// The larger of two candidates, the lower index of two equal ones.  NaN is never larger.
__device__ __forceinline__ void TakeLarger(float& best, int& idx, float v, int j)
{
  if (v > best || (v == best && j < idx)) {
    best = v;
    idx = j;
  }
}

// A cluster per row; the first index of the maximum wins (DxirInterpreter.kt:2414-2426).  The row is bound by latency, not by its bytes
// (32768 columns are 128 KB), so it is spread over up to eight CTAs whose threads have all their 16-byte loads in flight at once; one CTA a
// row, reading 128 elements a thread one after the other, took 30 us where this takes 4.
__global__ void __launch_bounds__(kArgmaxThreads) ArgmaxKernel(const float* x, int* out, int n, int per, int vec)
{
  GridDependencySync();
  constexpr int kWarps = kArgmaxThreads / 32, kUnroll = 8;
  __shared__ float bv[kWarps];
  __shared__ int bi[kWarps];
  __shared__ float cv[kArgmaxCluster];
  __shared__ int ci[kArgmaxCluster];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank()), ranks = static_cast<int>(cluster.num_blocks());
  const float* xr = x + static_cast<size_t>(blockIdx.x) * n;
  const int lo = rank * per, hi = min(n, lo + per), tid = threadIdx.x;
  float best = -INFINITY;
  int idx = 0x7fffffff;
  if (vec) {
    for (int j0 = lo + tid * 4; j0 < hi; j0 += kArgmaxThreads * 4 * kUnroll) {
      float4 v[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int j = j0 + u * kArgmaxThreads * 4;
        if (j < hi) v[u] = __ldcg(reinterpret_cast<const float4*>(xr + j));
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int j = j0 + u * kArgmaxThreads * 4;
        if (j < hi) {
          TakeLarger(best, idx, v[u].x, j);
          TakeLarger(best, idx, v[u].y, j + 1);
          TakeLarger(best, idx, v[u].z, j + 2);
          TakeLarger(best, idx, v[u].w, j + 3);
        }
      }
    }
  } else {
    for (int j = lo + tid; j < hi; j += kArgmaxThreads) TakeLarger(best, idx, xr[j], j);
  }
  const int lane = tid & 31, warp = tid >> 5;
  auto across = [&](int from) {
    for (int o = from; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      TakeLarger(best, idx, ov, oi);
    }
  };
  across(16);
  if (lane == 0) {
    bv[warp] = best;
    bi[warp] = idx;
  }
  __syncthreads();
  if (warp == 0) {
    best = lane < kWarps ? bv[lane] : -INFINITY;
    idx = lane < kWarps ? bi[lane] : 0x7fffffff;
    across(kWarps / 2);
  }
  if (ranks > 1) {
    cluster.sync();  // rank 0 runs: its shared memory may be written
    if (tid == 0) {
      cluster.map_shared_rank(cv, 0)[rank] = best;
      cluster.map_shared_rank(ci, 0)[rank] = idx;
    }
    cluster.sync();
    if (rank != 0) return;
    if (tid == 0) {
      for (int r = 1; r < ranks; ++r) TakeLarger(best, idx, cv[r], ci[r]);
    }
  }
  // A row of NaNs (or an empty comparison) leaves idx unset: the interpreter's answer is index 0.
  if (tid == 0) out[blockIdx.x] = idx == 0x7fffffff ? 0 : idx;
}

// The inputs of a step travel to the device as one copy and are handed out to their buffers here: each copy of its own costs about 5 us on the
// stream, and a step has five to eight of them.
constexpr int kMaxSegments = 16;
struct UnpackArgs {
  int32_t* dst[kMaxSegments];
  int start[kMaxSegments + 1];
  int segments;
};
__global__ void __launch_bounds__(256) UnpackKernel(const int32_t* packed, const __grid_constant__ UnpackArgs a)
{
  GridDependencySync();
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= a.start[a.segments]) return;
  int s = 0;
  while (i >= a.start[s + 1]) ++s;
  a.dst[s][i - a.start[s]] = __ldcg(packed + i);
}

template <typename TT>
cudaError_t LaunchEmbedding(const void* table, const int32_t* ids, float* out, int positions, int vocab, int dim, cudaStream_t st)
{
  constexpr int kPer = 16 / static_cast<int>(sizeof(TT));
  const dim3 grid(positions, std::min(65535, (dim - 1) / (kEmbedThreads * kPer) + 1));
  const TT* t = static_cast<const TT*>(table);
  return dim % kPer == 0 && Aligned16(table) && Aligned16(out) ? LaunchChained(EmbeddingKernel<TT, true>, grid, kEmbedThreads, 0, st, t, ids, out, vocab, dim)
                                                             : LaunchChained(EmbeddingKernel<TT, false>, grid, kEmbedThreads, 0, st, t, ids, out, vocab, dim);
}

}  // namespace
}  // namespace tlaloc_b200

using namespace tlaloc_b200;

extern "C" int tlaloc_b200_embedding(const void* table, int32_t table_dtype, const int32_t* ids, float* out,
                                     int32_t positions, int32_t vocab, int32_t dim, void* stream)
{
  if (!table || !ids || !out) return Fail(kInvalid, "EMBEDDING: a required device pointer is null");
  if (!IsFloatType(table_dtype)) return Fail(kInvalid, "EMBEDDING: the table must be f32 or bf16");
  if (positions < 0 || vocab < 1 || dim < 1) return Fail(kInvalid, "EMBEDDING: bad sizes");
  if (positions == 0) return kOk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const cudaError_t e = table_dtype == TLALOC_B200_F32 ? LaunchEmbedding<float>(table, ids, out, positions, vocab, dim, st)
                                                       : LaunchEmbedding<__nv_bfloat16>(table, ids, out, positions, vocab, dim, st);
  if (e != cudaSuccess) return CudaFail("EMBEDDING launch", e);
  CountLaunches(1);
  return kOk;
}

extern "C" int tlaloc_b200_argmax(const float* logits, int32_t* out, int32_t rows, int32_t n, void* stream)
{
  if (!logits || !out) return Fail(kInvalid, "ARGMAX: a required device pointer is null");
  if (rows < 0 || n < 1) return Fail(kInvalid, "ARGMAX: bad sizes");
  if (rows == 0) return kOk;
  // At least 4096 columns a CTA: two 16-byte loads per thread, below which another CTA costs more than it takes over.
  int ranks = 1;
  while (ranks < kArgmaxCluster && n >= ranks * 2 * 4096) ranks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(rows, ranks);
  cfg.blockDim = dim3(kArgmaxThreads);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cudaLaunchAttribute attrs[2];
  cfg.numAttrs = ChainAttributes(attrs, ranks);
  cfg.attrs = attrs;
  const int per = ((n + ranks - 1) / ranks + 3) / 4 * 4;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, ArgmaxKernel, logits, out, static_cast<int>(n), per, n % 4 == 0 && Aligned16(logits) ? 1 : 0);
  if (e != cudaSuccess) return CudaFail("ARGMAX launch", e);
  CountLaunches(1);
  return kOk;
}

extern "C" int tlaloc_b200_unpack_i32(const int32_t* packed, int32_t* const* dst, const int32_t* counts, int32_t segments, void* stream)
{
  if (!packed || !dst || !counts) return Fail(kInvalid, "UNPACK: a required pointer is null");
  if (segments < 1 || segments > kMaxSegments) return Fail(kInvalid, "UNPACK: 1 to %d segments", kMaxSegments);
  UnpackArgs a = {};
  a.segments = segments;
  long long total = 0;
  for (int i = 0; i < segments; ++i) {
    if (counts[i] < 0 || (counts[i] > 0 && !dst[i])) return Fail(kInvalid, "UNPACK: bad segment %d", i);
    a.dst[i] = dst[i];
    total += counts[i];
    if (total > (1 << 30)) return Fail(kInvalid, "UNPACK: too many values");
    a.start[i + 1] = static_cast<int>(total);
  }
  if (total == 0) return kOk;
  const cudaError_t e = LaunchChained(UnpackKernel, static_cast<unsigned>((total + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream), packed, a);
  if (e != cudaSuccess) return CudaFail("UNPACK launch", e);
  CountLaunches(1);
  return kOk;
}
