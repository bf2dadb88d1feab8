// The int8 weight-only projection y = (cast(x) @ cast(codes)) * scale for sm_100a
// (HfDecoderGraph.proj over WeightQuant.INT8, ir/.../inference/HfDecoderGraph.kt:625-655).
//
//   Int8GemvKernel   decode rows (M <= 32 per launch; by default only up to 16 rows come here, 17 and more go to the
//                    tensor-core kernels of int8_gemm_tc.cu and int8_gemm_i8.cu).  HBM-bound: every
//                    weight byte is read once, from the reference's own [K, N] layout (no repacking).  A CTA owns
//                    128 output columns and one slice of K; each of its four warps is an independent cp.async
//                    pipeline over its own 32-row stages (a 32 x 128 int8 weight tile plus the matching 32-wide
//                    strip of the bf16 activations, XOR-swizzled in shared memory), so there is no CTA-wide barrier
//                    in the loop and five CTAs fit an SM (one n-tile).  The MMA runs transposed: the 16 output columns a lane
//                    pair-set owns are the M dimension and the (<= 8 per n-tile) activation rows the N dimension, so
//                    one 16-row step costs 8 mma.sync m16n8k16 per n-tile.  The int8 codes become exact bf16 pairs in
//                    registers (one byte-permute, two logic ops and one packed bf16 add per pair); products are
//                    exact, accumulation fp32.  The K slices of one column tile form a thread-block cluster and are
//                    summed through distributed shared memory in rank order: no global scratch, no second kernel,
//                    and a result that does not depend on timing.  The per-column scale (and an optional residual)
//                    is applied to the finished sum, as the graph multiplies after the dot.
//                    Bound at one row by the issue of the conversion (ncu, 4096 x 28672: ALU pipe 57 %, issue slots 50 % busy, 3.3 warps a scheduler)
//                    and by the SMs that idle at its ends (22 % of the time).  4096 x 28672 with a norm in front: 34.3 us with two slices and a division
//                    per stage for the ring's place, 31.0 with three slices, 30.1 with places and sources that move on by themselves, 29.0 with the ranks' sums in flight together,
//                    27.1 with two stages a warp and five CTAs an SM in place of three and four.
//   GemmExactKernel  the interpreter's MATMUL order (DxirInterpreter.kt:739-765): f32, k ascending, separate
//                    multiply and add, zero activations skipped.  Bit-identical to the CPU oracle; slow.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace tlaloc_b200 {
namespace {

struct GemmParams {
  const __nv_bfloat16* x;  // [M, K] bf16
  const int8_t* w;         // [K, N]
  const float* scales;     // [N] or null
  const float* residual;   // [M, N] or null
  void* y;                 // [M, N]
  int M, K, N;
  int Kc;  // K per CTA (a multiple of kGvStageK * kGvWarps)
  int ks;  // K slices (cluster size along y)
  int weights_const;  // no kernel still in flight writes codes or scales: the first weight stages are fetched before the dependency wait
};

constexpr int kGvThreads = 128;
constexpr int kGvWarps = 4;
constexpr int kGvCols = 128;
constexpr int kGvStageK = 32;  // k rows per pipeline stage
constexpr int kGvWBytes = kGvStageK * kGvCols;  // the stage's weight tile
constexpr int kGvRedStride = kGvCols + 4;

__device__ __forceinline__ uint32_t SmemAddr(const void* ptr)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(ptr));
}
__device__ __forceinline__ void CpAsync16(uint32_t dst, const void* src, int src_bytes)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void CpAsyncCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void CpAsyncWait()
{
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void LdMatrixX2(uint32_t (&r)[2], uint32_t addr)
{
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ uint4 LdShared16(uint32_t addr)
{
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void MmaBf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Bytes `B` of two words (codes of two consecutive k for one column) as an exact bf16 pair, lower k in the low
// half.  For a code v with bits s:lo7, 0x4300|lo7 is the bf16 128 + lo7 and 0xC300|s<<7 is -128 or -256; their
// sum is v, exactly.
template <int B>
__device__ __forceinline__ uint32_t CodesToBf16x2(uint32_t w_lo_k, uint32_t w_hi_k)
{
  const uint32_t q = __byte_perm(w_lo_k, w_hi_k, B | (B << 4) | ((4 + B) << 8) | ((4 + B) << 12));
  uint32_t t, c;  // (q & mask) | magic as one three-input logic op each
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(t) : "r"(q), "r"(0x007F007Fu), "r"(0x43004300u));
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;\n" : "=r"(c) : "r"(q), "r"(0x00800080u), "r"(0xC300C300u));
  uint32_t r;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;\n" : "=r"(r) : "r"(t), "r"(0x3F803F80u), "r"(c));
  return r;
}

// NT: n-tiles of eight activation rows.  S: stages of a warp.  Registers allow five CTAs an SM with one n-tile (96 a thread) and four with two (126); three stages leave room in
// shared memory for four and three.  (Six CTAs, by a bound of 80 registers and 16 bytes of spills: 4096 x 14336 at one row 16.4 -> 20.0 us, 4096 x 4096 6.6 -> 7.0.)
// LaunchGemv says which is taken where.
template <int NT, int S>
struct GvLayout {
  static constexpr int kRows = NT * 8;                     // activation rows a launch covers
  static constexpr int kXBytes = kRows * kGvStageK * 2;    // the stage's activation strip, [rows][32] bf16
  static constexpr int kStageBytes = kGvWBytes + kXBytes;
  static constexpr int kWarpBytes = S * kStageBytes;
  static constexpr int kPipeBytes = kGvWarps * kWarpBytes;
  // After the loop the same space holds the four warps' partial tiles and the CTA's summed tile.
  static constexpr int kTileBytes = kRows * kGvRedStride * 4;
  static constexpr int kRedBytes = (kGvWarps + 1) * kTileBytes;
  static constexpr int kBytes = kPipeBytes > kRedBytes ? kPipeBytes : kRedBytes;
};

template <int NT, int S, typename YT>
__global__ void __launch_bounds__(kGvThreads) Int8GemvKernel(GemmParams p)
{
  if (!p.weights_const) GridDependencySync();
  using L = GvLayout<NT, S>;
  extern __shared__ __align__(128) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int col0 = blockIdx.x * kGvCols;
  const int kb = blockIdx.y * p.Kc;
  const int ke = min(p.K, kb + p.Kc);
  const int nstages = ke > kb ? (ke - kb + kGvStageK - 1) / kGvStageK : 0;
  const int my_n = warp < nstages ? (nstages - warp + kGvWarps - 1) / kGvWarps : 0;
  const uint32_t my_pipe_addr = SmemAddr(smem + warp * L::kWarpBytes);

  // Copies of one stage (k rows [k0, k0 + 32) of this warp), all lane-invariant parts computed once.
  //   weights: copy i of lane (l3 = lane >> 3, ch = lane & 7) moves row l3 + 4i, 16-byte chunk ch, to chunk
  //            ch ^ (row & 6): (row & 6) is (l3 & 2) for even i and (l3 & 2) | 4 for odd i;
  //   activations: copy i moves row (lane >> 2) + 8i, 16-byte piece lane & 3, to piece ^ ((row >> 1) & 3).
  // The reads further down are then conflict-free.  K is a multiple of 8 and N of 16 on this path, so a chunk is
  // wholly inside or outside the matrix; outside is zero-filled.
  const int l3 = lane >> 3, ch = lane & 7;
  const bool col_ok = col0 + ch * 16 < p.N;
  const uint32_t wdst_even = l3 * kGvCols + ((ch ^ (l3 & 2)) << 4);
  const uint32_t wdst_odd = (l3 + 4) * kGvCols + ((ch ^ ((l3 & 2) | 4)) << 4);
  const size_t w_row4 = static_cast<size_t>(4) * p.N;
  const int8_t* w_lane = p.w + static_cast<size_t>(kb + warp * kGvStageK + l3) * p.N + col0 + (col_ok ? ch * 16 : 0);
  const size_t w_stage = static_cast<size_t>(kGvWarps * kGvStageK) * p.N;
  const int xm = lane >> 2, xpiece = lane & 3;
  const uint32_t xdst = kGvWBytes + xm * (kGvStageK * 2) + ((xpiece ^ ((xm >> 1) & 3)) << 4);
  const __nv_bfloat16* x_lane = p.x + static_cast<size_t>(xm) * p.K + kb + warp * kGvStageK + xpiece * 8;

  // A stage's copies in two parts: the weights, which with weights_const depend on no earlier kernel, and the activations.  Both go through the
  // slice from front to back; the ring's place and the sources move on by themselves, without a division or a product per stage.
  int w_k0 = kb + warp * kGvStageK, x_k0 = w_k0;
  uint32_t w_place = my_pipe_addr, x_place = my_pipe_addr;
  const uint32_t ring_end = my_pipe_addr + L::kWarpBytes;
  auto issue_w = [&]() {
    if (w_k0 + kGvStageK <= ke) {  // the whole stage is inside K
      const int bytes = col_ok ? 16 : 0;
#pragma unroll
      for (int i = 0; i < 8; i += 2) {
        CpAsync16(w_place + wdst_even + i * (4 * kGvCols), w_lane + i * w_row4, bytes);
        CpAsync16(w_place + wdst_odd + i * (4 * kGvCols), w_lane + (i + 1) * w_row4, bytes);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool valid = col_ok && w_k0 + l3 + 4 * i < ke;
        CpAsync16(w_place + ((i & 1) ? wdst_odd - 4 * kGvCols : wdst_even) + i * (4 * kGvCols), valid ? w_lane + i * w_row4 : p.w, valid ? 16 : 0);
      }
    }
    w_k0 += kGvWarps * kGvStageK;
    w_lane += w_stage;
    w_place = w_place + L::kStageBytes == ring_end ? my_pipe_addr : w_place + L::kStageBytes;
  };
  auto issue_x = [&]() {
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const bool valid = xm + 8 * i < p.M && x_k0 + xpiece * 8 < ke;
      CpAsync16(x_place + xdst + i * (8 * kGvStageK * 2), valid ? x_lane + static_cast<size_t>(8 * i) * p.K : p.x, valid ? 16 : 0);
    }
    x_k0 += kGvWarps * kGvStageK;
    x_lane += kGvWarps * kGvStageK;
    x_place = x_place + L::kStageBytes == ring_end ? my_pipe_addr : x_place + L::kStageBytes;
  };

  if (p.weights_const) {
    // The weights of the first stages are on their way while the previous kernel drains; the first commit group then
    // holds all of them together with the first stage's activations.
    for (int it = 0; it < S - 1; ++it)
      if (it < my_n) issue_w();
    GridDependencySync();
    for (int it = 0; it < S - 1; ++it) {
      if (it < my_n) issue_x();
      CpAsyncCommit();
    }
  } else {
    for (int it = 0; it < S - 1; ++it) {
      if (it < my_n) {
        issue_w();
        issue_x();
      }
      CpAsyncCommit();
    }
  }

  // acc[j][nt]: output columns col0 + gid*16 + 2j (c0, c1) and + 2j + 1 (c2, c3), activation rows nt*8 + 2tig, + 1.
  float acc[8][NT][4];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) acc[j][nt][0] = acc[j][nt][1] = acc[j][nt][2] = acc[j][nt][3] = 0.f;

  // Reads of a stage.  Weights: this lane's 16 columns (chunk gid) of rows 2tig + {0, 1, 8, 9} of each 16-row step;
  // for all of them (row & 6) == 2tig.  Activations (ldmatrix): row lane & 7 of the n-tile, piece 2h + ((lane >> 3) & 1).
  const uint32_t wread = (2 * tig) * kGvCols + ((gid ^ (2 * tig)) << 4);
  const int xr = lane & 7, xsw = (xr >> 1) & 3, xp0 = (lane >> 3) & 1;
  const uint32_t xread0 = kGvWBytes + xr * (kGvStageK * 2) + ((xp0 ^ xsw) << 4);
  const uint32_t xread1 = kGvWBytes + xr * (kGvStageK * 2) + (((xp0 + 2) ^ xsw) << 4);

  uint32_t st_addr = my_pipe_addr;
  for (int it = 0; it < my_n; ++it) {
    if (it + S - 1 < my_n) {
      issue_w();
      issue_x();
    }
    CpAsyncCommit();
    CpAsyncWait<S - 1>();
    __syncwarp();
#pragma unroll
    for (int h = 0; h < kGvStageK / 16; ++h) {
      // x^T as B fragments: b0b1 = x[row gid][16h + 2tig, +1], b2b3 = x[row gid][16h + 8 + 2tig, +1].
      uint32_t b[NT][2];
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) LdMatrixX2(b[nt], st_addr + (h ? xread1 : xread0) + nt * (8 * kGvStageK * 2));
      const uint32_t wbase = st_addr + wread + h * (16 * kGvCols);
      const uint4 ra = LdShared16(wbase), rb = LdShared16(wbase + kGvCols);
      const uint4 rc = LdShared16(wbase + 8 * kGvCols), rd = LdShared16(wbase + 9 * kGvCols);
      const uint32_t wa[4] = {ra.x, ra.y, ra.z, ra.w}, wb[4] = {rb.x, rb.y, rb.z, rb.w};
      const uint32_t wc[4] = {rc.x, rc.y, rc.z, rc.w}, wd[4] = {rd.x, rd.y, rd.z, rd.w};
#pragma unroll
      for (int wi = 0; wi < 4; ++wi) {
        // Bytes 0, 1 of word wi are columns 4wi, 4wi + 1 (MMA j = 2wi); bytes 2, 3 are MMA j = 2wi + 1.
        uint32_t a0[4], a1[4];
        a0[0] = CodesToBf16x2<0>(wa[wi], wb[wi]);
        a0[1] = CodesToBf16x2<1>(wa[wi], wb[wi]);
        a0[2] = CodesToBf16x2<0>(wc[wi], wd[wi]);
        a0[3] = CodesToBf16x2<1>(wc[wi], wd[wi]);
        a1[0] = CodesToBf16x2<2>(wa[wi], wb[wi]);
        a1[1] = CodesToBf16x2<3>(wa[wi], wb[wi]);
        a1[2] = CodesToBf16x2<2>(wc[wi], wd[wi]);
        a1[3] = CodesToBf16x2<3>(wc[wi], wd[wi]);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          MmaBf16(acc[2 * wi][nt], a0, b[nt][0], b[nt][1]);
          MmaBf16(acc[2 * wi + 1][nt], a1, b[nt][0], b[nt][1]);
        }
      }
    }
    __syncwarp();  // the stage is free for the copy the next iteration issues
    st_addr = st_addr + L::kStageBytes == ring_end ? my_pipe_addr : st_addr + L::kStageBytes;
  }
  CpAsyncWait<0>();
  __syncthreads();  // every warp is done with the pipeline space

  // The four warps' partial tiles -> shared memory -> one tile, summed in warp order.
  float* red = reinterpret_cast<float*>(smem);                  // [kGvWarps][kRows][kGvRedStride]
  float* tile = red + kGvWarps * (L::kRows * kGvRedStride);     // [kRows][kGvRedStride]
  {
    float* mine = red + warp * (L::kRows * kGvRedStride);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int m = nt * 8 + 2 * tig, c = gid * 16 + 2 * j;
        mine[m * kGvRedStride + c] = acc[j][nt][0];
        mine[(m + 1) * kGvRedStride + c] = acc[j][nt][1];
        mine[m * kGvRedStride + c + 1] = acc[j][nt][2];
        mine[(m + 1) * kGvRedStride + c + 1] = acc[j][nt][3];
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < p.M * kGvCols; e += kGvThreads) {
    const int m = e / kGvCols, c = e - m * kGvCols;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < kGvWarps; ++w) v += red[w * (L::kRows * kGvRedStride) + m * kGvRedStride + c];
    tile[m * kGvRedStride + c] = v;
  }
  // The K slices of this column tile are the ranks of one cluster: rank r finishes every ks-th row.
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), nranks = cluster.num_blocks();
  const int col = col0 + tid;
  const float scale = p.scales != nullptr && col < p.N ? __ldg(p.scales + col) : 1.f;  // on its way while the ranks meet
  cluster.sync();
  YT* y = static_cast<YT*>(p.y);
  constexpr int kU = NT == 1 ? 1 : 2;  // rows at a time: with eight ranks a CTA has one of eight rows, two of sixteen
  for (int m0 = rank; m0 < p.M && col < p.N; m0 += kU * nranks) {
    float v[kU], residual[kU];
#pragma unroll
    for (int e = 0; e < kU; ++e) {
      const int m = m0 + e * static_cast<int>(nranks);
      residual[e] = p.residual != nullptr && m < p.M ? __ldg(p.residual + static_cast<size_t>(m) * p.N + col) : 0.f;
    }
    SumRanks(tile + m0 * kGvRedStride + tid, nranks, nranks * kGvRedStride, (p.M - m0 + nranks - 1) / nranks, v);
#pragma unroll
    for (int e = 0; e < kU; ++e) {
      const int m = m0 + e * static_cast<int>(nranks);
      if (m >= p.M) break;
      if (p.scales != nullptr) v[e] *= scale;
      if (p.residual != nullptr) v[e] += residual[e];
      y[static_cast<size_t>(m) * p.N + col] = FromF32<YT>(v[e]);
    }
  }
  cluster.sync();  // no CTA leaves while a peer may still read its tile
}

// ------------------------------------------------------------------------------------------

// Eight values a thread (n is a multiple of eight here: k is), by 16-byte words where x allows.
__global__ void __launch_bounds__(256) ToBf16Kernel(const float* x, __nv_bfloat16* out, size_t n, int vec)
{
  GridDependencySync();
  const size_t i = (static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x) * 8;
  if (i >= n) return;
  float v[8];
  if (vec) {
    *reinterpret_cast<float4*>(v) = __ldcg(reinterpret_cast<const float4*>(x + i));
    *reinterpret_cast<float4*>(v + 4) = __ldcg(reinterpret_cast<const float4*>(x + i) + 1);
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = x[i + e];
  }
  uint4 o;
  uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    w[e] = *reinterpret_cast<const uint32_t*>(&b);
  }
  *reinterpret_cast<uint4*>(out + i) = o;
}
cudaError_t LaunchToBf16(const void* x, void* out, size_t count, cudaStream_t st)
{
  return LaunchChained(ToBf16Kernel, static_cast<unsigned>((count / 8 + 255) / 256), 256, 0, st, static_cast<const float*>(x), static_cast<__nv_bfloat16*>(out),
                       count, Aligned16(x) ? 1 : 0);
}

// y[i, j] = (sum over p ascending of x[i, p] * w[p, j], f32, separate multiply and add, x == 0 skipped) * scale[j]
// (+ residual).  Grid (ceil(N / 256), M).
template <typename XT, typename WT, typename YT>
__global__ void __launch_bounds__(256) GemmExactKernel(const XT* x, const WT* w, const float* scales,
                                                       const float* residual, YT* y, int M, int K, int N,
                                                       int round_x)
{
  GridDependencySync();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  if (j >= N) return;
  float acc = 0.f;
  for (int p = 0; p < K; ++p) {
    float a = ToF32(x[static_cast<size_t>(i) * K + p]);
    if (round_x) a = __bfloat162float(__float2bfloat16_rn(a));
    if (a == 0.f) continue;
    acc = __fadd_rn(acc, __fmul_rn(a, ToF32(w[static_cast<size_t>(p) * N + j])));
  }
  if (scales != nullptr) acc = __fmul_rn(acc, scales[j]);
  if (residual != nullptr) acc = __fadd_rn(acc, residual[static_cast<size_t>(i) * N + j]);
  y[static_cast<size_t>(i) * N + j] = FromF32<YT>(acc);
}

// The fused gate|up projection + SwiGLU in the interpreter's order, for shapes the tensor-core kernel does not take:
// column j of the result reads gate column (j / 128) * 256 + j % 128 and up column 128 further on.
template <typename XT, typename YT>
__global__ void __launch_bounds__(256) GemmSwigluExactKernel(const XT* x, const int8_t* w, const float* scales, YT* y, int M, int K,
                                                             int N, int round_x, int faithful)
{
  GridDependencySync();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  const int half = N >> 1;
  if (j >= half) return;
  const int cg = (j >> 7) * 256 + (j & 127), cu = cg + 128;
  float g = 0.f, u = 0.f;
  for (int p = 0; p < K; ++p) {
    float a = ToF32(x[static_cast<size_t>(i) * K + p]);
    if (round_x) a = __bfloat162float(__float2bfloat16_rn(a));
    if (a == 0.f) continue;
    g = __fadd_rn(g, __fmul_rn(a, ToF32(w[static_cast<size_t>(p) * N + cg])));
    u = __fadd_rn(u, __fmul_rn(a, ToF32(w[static_cast<size_t>(p) * N + cu])));
  }
  if (scales != nullptr) {
    g = __fmul_rn(g, scales[cg]);
    u = __fmul_rn(u, scales[cu]);
  }
  float silu;
  if (faithful) {
    const double gd = static_cast<double>(g);
    silu = static_cast<float>(gd / (1.0 + exp(-gd)));
  } else {
    silu = g / (1.f + expf(-g));
  }
  y[static_cast<size_t>(i) * half + j] = FromF32<YT>(__fmul_rn(silu, u));
}

template <int NT, typename YT>
cudaError_t PrepareGemv()
{
  const cudaError_t e = cudaFuncSetAttribute(Int8GemvKernel<NT, 2, YT>, cudaFuncAttributeMaxDynamicSharedMemorySize, GvLayout<NT, 2>::kBytes);
  return e != cudaSuccess ? e : cudaFuncSetAttribute(Int8GemvKernel<NT, 3, YT>, cudaFuncAttributeMaxDynamicSharedMemorySize, GvLayout<NT, 3>::kBytes);
}

template <int NT, int S, typename YT>
cudaError_t LaunchGemvStages(const GemmParams& p, cudaStream_t stream)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((p.N + kGvCols - 1) / kGvCols, p.ks, 1);
  cfg.blockDim = dim3(kGvThreads, 1, 1);
  cfg.dynamicSmemBytes = GvLayout<NT, S>::kBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  cfg.numAttrs = ChainAttributes(attr, p.ks);
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, Int8GemvKernel<NT, S, YT>, p);
}
constexpr int kSms = 148;
template <int NT, typename YT>
cudaError_t LaunchGemv(const GemmParams& p, cudaStream_t stream)
{
  const int ctas = (p.N + kGvCols - 1) / kGvCols * p.ks;
  const int slice = (p.K + p.ks - 1) / p.ks;
  constexpr int kUnit = kGvStageK * kGvWarps;
  // Three stages where a third hides more than a fifth (NT 2: a fourth) CTA an SM would, us with two and three:
  //   NT 1  one CTA an SM: 1 row of 8192 x 1024 6.6, 6.2.  A full SM of long slices: 4096 x 32768 (512 CTAs of 2048 k) 29.9, 25.0, 28672 x 8192 50.2, 41.3, either the
  //         same behind a norm.  Not shorter ones: 2048 x 8192 (512 of 256 k) behind a norm 7.8, 8.9; nor between: 5120 x 5120 (320) 8.6, 9.9; nor more CTAs: 4096 x 28672 (672) 22.5, 24.8.
  //   NT 2  up to what three CTAs an SM hold in one wave of clusters: 9 rows of 4096 x 6144 (384) 10.7, 9.4, 5120 x 5120 (320) 12.2, 10.5, a step of 12 rows through three 8B-shape layers
  //         403, 390; but 2560 x 11008 in 430 11.0, 13.8, 28672 x 8192 in 512 49.2, 60.8, 12 rows through two 70B-shape layers 594 with three there, 551 with two.
  //         Far more CTAs of long slices again: the same 8B-shape step, its 4096 x 28672 (672 of 1366 k) with two 399, with three 389.
  const bool three = NT == 1 ? ctas <= kSms || (ctas > 3 * kSms && ctas <= 4 * kSms && slice >= 16 * kUnit)
                             : 5 * ctas <= 13 * kSms || (ctas > 4 * kSms && slice >= 10 * kUnit);
  return three ? LaunchGemvStages<NT, 3, YT>(p, stream) : LaunchGemvStages<NT, 2, YT>(p, stream);
}

// K slices for a shape, one to eight (the portable cluster sizes; not seven, which came out slower than six and eight wherever measured).  What counts is how evenly
// the CTAs fall on the 148 SMs and that there are about three an SM, so that loads in flight cover the way to HBM, and how much of the longest slice the average one has; more slices
// than that have to be worth a seventh.  Columns that are cut
// evenly over all SMs instead (112 or 96 a CTA) lose more to rows of codes that start within a 128-byte line than the last wave costs.
// Microseconds at one row with a norm in front, slices 2 / 3 / 4 of 4096 x 28672: 30.1 / 27.4 / 30.5; 4 / 5 / 6 of 5120 x 14336: 21.2 / 19.0 / 20.0;
// 4 / 6 / 8 of 14336 x 4096: 20.9 / 19.8 / 16.5.  Not taken are
//   a slice without rows (2560 in eight is seven of 384: 2560 x 8192 at one row 8.5, 7.0 in four),
//   beyond two CTAs an SM a slice of less than four stages a warp, whose beginning and end outweigh it (2048 x 8192 at 8 rows 8.0 in eight, 7.1 in four), unless k has no more to begin with,
//   a second wave (five CTAs an SM up to 8 rows, four from 9 on) of less than nine (4096 x 11008 in eight: 1 row 11.0, 9 rows 17.1, in six 13.6, 14.4).
// $TLALOC_B200_GEMV_KS overrides.
int ChooseSlices(int k, int n, int rows)
{
  static const int forced = [] {
    const char* e = std::getenv("TLALOC_B200_GEMV_KS");
    return e != nullptr ? std::atoi(e) : 0;
  }();
  if (forced >= 1 && forced <= 8) return forced;
  constexpr int kWanted = 3 * kSms;
  const int tiles = (n + kGvCols - 1) / kGvCols;
  int best = 1;
  double best_score = 0.0;
  for (int ks = 1; ks <= 8; ++ks) {
    if (ks > 1 && k / ks < kGvStageK * kGvWarps) break;
    if (ks == 7) continue;
    const int items = tiles * ks, share = (items + kSms - 1) / kSms;
    const int unit = kGvStageK * kGvWarps, slice = ((k + ks - 1) / ks + unit - 1) / unit * unit;
    if (ks > 1 && slice * (ks - 1) >= k) continue;
    if (ks > 1 && items > 2 * kSms && slice < 4 * unit && k >= 4 * unit) continue;
    if (ks > 1 && items > (rows > 8 ? 4 : 5) * kSms && slice <= 8 * unit) continue;
    const double score = static_cast<double>(items) / (share * kSms) * std::min(1.0, static_cast<double>(items) / kWanted) * k / (static_cast<double>(ks) * slice);
    if (score > best_score * (tiles * best < kWanted ? 1.08 : 1.15)) {
      best_score = score;
      best = ks;
    }
  }
  return best;
}

}  // namespace

cudaError_t PrepareInt8GemmKernels()
{
  static OncePerDevice once;
  return once.Run([](int) {
    cudaError_t e = PrepareGemv<1, float>();
    if (e == cudaSuccess) e = PrepareGemv<1, __nv_bfloat16>();
    if (e == cudaSuccess) e = PrepareGemv<2, float>();
    if (e == cudaSuccess) e = PrepareGemv<2, __nv_bfloat16>();
    if (e == cudaSuccess) e = PrepareGemv<4, float>();
    if (e == cudaSuccess) e = PrepareGemv<4, __nv_bfloat16>();
    return e;
  });
}
namespace {
KernelSetup g_setup(PrepareInt8GemmKernels, nullptr);
}

}  // namespace tlaloc_b200

using namespace tlaloc_b200;

namespace {

bool FastShape(int k, int n) { return n % 16 == 0 && k % 8 == 0 && k >= 16; }

template <typename XT, typename WT>
cudaError_t LaunchExact(const void* x, const void* w, const float* scales, const float* residual, void* y,
                        int y_dtype, int m, int k, int n, int round_x, cudaStream_t st)
{
  const dim3 grid((n + 255) / 256, m);
  if (y_dtype == TLALOC_B200_F32) {
    return LaunchChained(GemmExactKernel<XT, WT, float>, grid, 256, 0, st, static_cast<const XT*>(x),
                         static_cast<const WT*>(w), scales, residual, static_cast<float*>(y), m, k, n, round_x);
  }
  return LaunchChained(GemmExactKernel<XT, WT, __nv_bfloat16>, grid, 256, 0, st, static_cast<const XT*>(x),
                       static_cast<const WT*>(w), scales, residual, static_cast<__nv_bfloat16*>(y), m, k, n, round_x);
}

template <typename YT>
cudaError_t LaunchGemvRows(const GemmParams& p, int rows, cudaStream_t st)
{
  if (rows <= 8) return LaunchGemv<1, YT>(p, st);
  if (rows <= 16) return LaunchGemv<2, YT>(p, st);
  return LaunchGemv<4, YT>(p, st);
}

}  // namespace

// Scratch: the bf16 copy of an f32 x, or the two int8 planes of the activations and their row steps.
extern "C" size_t tlaloc_b200_int8_gemm_scratch_bytes(int32_t m, int32_t k, int32_t n)
{
  (void)n;
  if (m <= 0 || k <= 0) return 0;
  return (Int8GemmI8ScratchBytes(m, k) + 255) / 256 * 256;
}

namespace {
int TcMinRows()
{
  static const int tc_min = [] {
    const char* v = std::getenv("TLALOC_B200_GEMM_TC_MIN");
    return v != nullptr ? std::atoi(v) : 17;
  }();
  return tc_min;
}
// 17 to 128 rows, the caller's consent and room in the scratch: the int8 tensor-core kernel.
bool UseI8(const int8_t* codes, const void* scratch, size_t scratch_bytes, int m, int k, int n, int flags)
{
  return (flags & TLALOC_B200_GEMM_I8_MMA) != 0 && m >= TcMinRows() && Int8GemmI8Applies(codes, m, k, n) && scratch != nullptr && Aligned16(scratch) &&
         scratch_bytes >= Int8GemmI8ScratchBytes(m, k);
}
}  // namespace

extern "C" int tlaloc_b200_int8_gemm(const void* x, int32_t x_dtype, const int8_t* codes, const float* scales,
                                     const float* residual, void* y, int32_t y_dtype, float* scratch,
                                     size_t scratch_bytes, int32_t m, int32_t k, int32_t n, int32_t flags,
                                     void* stream)
{
  const char* op = "INT8_PROJ";
  if (!x || !codes || !y) return Fail(kInvalid, "%s: a required device pointer is null", op);
  if (!IsFloatType(x_dtype) || !IsFloatType(y_dtype)) return Fail(kInvalid, "%s: x and y must be f32 or bf16", op);
  if (m < 1 || k < 1 || n < 1) return Fail(kInvalid, "%s: needs positive [M, K] x [K, N], got M %d K %d N %d", op, m, k, n);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  // The fast kernels move x and the codes in 16-byte pieces: a view that starts off a 16-byte boundary (x + 4 elements,
  // a weight slice at an odd column) takes the order-faithful kernel instead, which has no alignment needs.
  const bool aligned = Aligned16(codes) && (x_dtype == TLALOC_B200_F32 || Aligned16(x));
  if ((flags & TLALOC_B200_GEMM_EXACT) != 0 || OrderFaithful() || !FastShape(k, n) || !aligned) {
    const int round_x = x_dtype == TLALOC_B200_F32 && (flags & TLALOC_B200_GEMM_X_F32_EXACT) == 0;
    e = x_dtype == TLALOC_B200_F32
            ? LaunchExact<float, int8_t>(x, codes, scales, residual, y, y_dtype, m, k, n, round_x, st)
            : LaunchExact<__nv_bfloat16, int8_t>(x, codes, scales, residual, y, y_dtype, m, k, n, 0, st);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ exact launch", e);
    CountLaunches(1);
    return kOk;
  }
  e = PrepareInt8GemmKernels();
  if (e != cudaSuccess) return CudaFail("INT8_PROJ set-up", e);
  if (UseI8(codes, scratch, scratch_bytes, m, k, n, flags)) {
    int launches = 0;
    e = LaunchInt8GemmI8(x, x_dtype, codes, scales, residual, y, y_dtype, scratch, m, k, n, st, &launches,
                         (flags & TLALOC_B200_GEMM_WEIGHTS_CONST) != 0, false, (flags & TLALOC_B200_GEMM_X_PLANES) != 0);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ int8 tensor-core launch", e);
    CountLaunches(launches);
    return kOk;
  }
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  if (x_dtype == TLALOC_B200_F32) {
    const size_t need = sizeof(__nv_bfloat16) * static_cast<size_t>(m) * k;
    if (scratch == nullptr || scratch_bytes < need) {
      return Fail(kInvalid, "%s: an f32 x needs %zu bytes of scratch for its bf16 copy, got %zu", op, need, scratch_bytes);
    }
    if (!Aligned16(scratch)) return Fail(kInvalid, "%s: scratch must be 16-byte aligned", op);
    const size_t count = static_cast<size_t>(m) * k;
    e = LaunchToBf16(x, scratch, count, st);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ activation cast", e);
    CountLaunches(1);
    xb = reinterpret_cast<const __nv_bfloat16*>(scratch);
  }
  const int tc_min = TcMinRows();
  // 17 rows and more: the tcgen05 kernel (measured at 32 rows: 123 vs 193 us at 57344 x 8192, 190 vs 216 us at the
  // 128256 x 4096 head; at 17 rows 166 vs 198 us; at 8 rows the row-vector kernel is faster, 103 vs ~165 us)
  if (m >= tc_min) {
    e = PrepareInt8GemmTcKernels();
    if (e != cudaSuccess) return CudaFail("INT8_PROJ set-up", e);
    int launches = 0;
    e = LaunchInt8GemmTc(xb, codes, scales, residual, y, y_dtype, m, k, n, st, &launches,
                         (flags & TLALOC_B200_GEMM_WEIGHTS_CONST) != 0);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ tensor-core launch", e);
    CountLaunches(launches);
    return kOk;
  }
  GemmParams p;
  p.w = codes;
  p.scales = scales;
  p.K = k;
  p.N = n;
  p.ks = ChooseSlices(k, n, m);
  p.weights_const = (flags & TLALOC_B200_GEMM_WEIGHTS_CONST) != 0 ? 1 : 0;
  const int per = (k + p.ks - 1) / p.ks;
  const int unit = kGvStageK * kGvWarps;
  p.Kc = (per + unit - 1) / unit * unit;
  const size_t ybytes = DtypeBytes(y_dtype);
  for (int m0 = 0; m0 < m; m0 += 32) {
    const int rows = std::min(32, m - m0);
    p.M = rows;
    p.x = xb + static_cast<size_t>(m0) * k;
    p.residual = residual ? residual + static_cast<size_t>(m0) * n : nullptr;
    p.y = static_cast<unsigned char*>(y) + static_cast<size_t>(m0) * n * ybytes;
    e = y_dtype == TLALOC_B200_F32 ? LaunchGemvRows<float>(p, rows, st) : LaunchGemvRows<__nv_bfloat16>(p, rows, st);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ launch", e);
    CountLaunches(1);
  }
  return kOk;
}

extern "C" int tlaloc_b200_dense_gemm_exact(const void* x, int32_t x_dtype, const void* w, int32_t w_dtype, float* y,
                                            int32_t m, int32_t k, int32_t n, int32_t flags, void* stream)
{
  const char* op = "MATMUL";
  if (!x || !w || !y) return Fail(kInvalid, "%s: a required device pointer is null", op);
  if (!IsFloatType(x_dtype) || !IsFloatType(w_dtype)) return Fail(kInvalid, "%s: x and w must be f32 or bf16", op);
  if (m < 1 || k < 1 || n < 1) return Fail(kInvalid, "%s: needs positive [M, K] x [K, N], got M %d K %d N %d", op, m, k, n);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // An f32 x meets a bf16 weight as bf16 (HfDecoderGraph.kt:641-647) unless the caller keeps it f32.
  const int round_x = x_dtype == TLALOC_B200_F32 && w_dtype == TLALOC_B200_BF16 && (flags & TLALOC_B200_GEMM_X_F32_EXACT) == 0;
  cudaError_t e;
  if (x_dtype == TLALOC_B200_F32 && w_dtype == TLALOC_B200_F32) {
    e = LaunchExact<float, float>(x, w, nullptr, nullptr, y, TLALOC_B200_F32, m, k, n, 0, st);
  } else if (x_dtype == TLALOC_B200_F32) {
    e = LaunchExact<float, __nv_bfloat16>(x, w, nullptr, nullptr, y, TLALOC_B200_F32, m, k, n, round_x, st);
  } else if (w_dtype == TLALOC_B200_F32) {
    e = LaunchExact<__nv_bfloat16, float>(x, w, nullptr, nullptr, y, TLALOC_B200_F32, m, k, n, 0, st);
  } else {
    e = LaunchExact<__nv_bfloat16, __nv_bfloat16>(x, w, nullptr, nullptr, y, TLALOC_B200_F32, m, k, n, 0, st);
  }
  if (e != cudaSuccess) return CudaFail("MATMUL exact launch", e);
  CountLaunches(1);
  return kOk;
}

extern "C" int tlaloc_b200_int8_gemm_swiglu(const void* x, int32_t x_dtype, const int8_t* codes, const float* scales, void* y,
                                            int32_t y_dtype, float* scratch, size_t scratch_bytes, int32_t m, int32_t k, int32_t n,
                                            int32_t flags, void* stream)
{
  const char* op = "INT8_PROJ_SWIGLU";
  if (!x || !codes || !y) return Fail(kInvalid, "%s: a required device pointer is null", op);
  if (!IsFloatType(x_dtype) || !IsFloatType(y_dtype)) return Fail(kInvalid, "%s: x and y must be f32 or bf16", op);
  if (m < 1 || k < 1 || n < 256 || n % 256 != 0) {
    return Fail(kInvalid, "%s: needs [M, K] x [K, N] with N a multiple of 256 (gate|up blocks of 128 + 128), got M %d K %d N %d", op, m, k, n);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int tc_min = TcMinRows();
  const bool aligned = Aligned16(codes) && (x_dtype == TLALOC_B200_F32 || Aligned16(x)) && (reinterpret_cast<uintptr_t>(y) & 7) == 0;
  cudaError_t e;
  if ((flags & TLALOC_B200_GEMM_EXACT) != 0 || OrderFaithful() || !FastShape(k, n) || !aligned || m < tc_min) {
    const int faithful = (flags & TLALOC_B200_GEMM_EXACT) != 0 || OrderFaithful();
    const int round_x = x_dtype == TLALOC_B200_F32 && (flags & TLALOC_B200_GEMM_X_F32_EXACT) == 0;
    const dim3 grid((n / 2 + 255) / 256, m);
#define TLALOC_SWIGLU_EXACT(XT, YT, RX)                                                                                  \
  e = LaunchChained(GemmSwigluExactKernel<XT, YT>, grid, 256, 0, st, static_cast<const XT*>(x), codes, scales,         \
                    static_cast<YT*>(y), m, k, n, RX, faithful)
    if (x_dtype == TLALOC_B200_F32 && y_dtype == TLALOC_B200_F32) TLALOC_SWIGLU_EXACT(float, float, round_x);
    else if (x_dtype == TLALOC_B200_F32) TLALOC_SWIGLU_EXACT(float, __nv_bfloat16, round_x);
    else if (y_dtype == TLALOC_B200_F32) TLALOC_SWIGLU_EXACT(__nv_bfloat16, float, 0);
    else TLALOC_SWIGLU_EXACT(__nv_bfloat16, __nv_bfloat16, 0);
#undef TLALOC_SWIGLU_EXACT
    if (e != cudaSuccess) return CudaFail("INT8_PROJ_SWIGLU exact launch", e);
    CountLaunches(1);
    return kOk;
  }
  if (UseI8(codes, scratch, scratch_bytes, m, k, n, flags)) {
    int launches = 0;
    e = LaunchInt8GemmI8(x, x_dtype, codes, scales, nullptr, y, y_dtype, scratch, m, k, n, st, &launches,
                         (flags & TLALOC_B200_GEMM_WEIGHTS_CONST) != 0, true, (flags & TLALOC_B200_GEMM_X_PLANES) != 0);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ_SWIGLU int8 tensor-core launch", e);
    CountLaunches(launches);
    return kOk;
  }
  const __nv_bfloat16* xb = static_cast<const __nv_bfloat16*>(x);
  if (x_dtype == TLALOC_B200_F32) {
    const size_t need = sizeof(__nv_bfloat16) * static_cast<size_t>(m) * k;
    if (scratch == nullptr || scratch_bytes < need || !Aligned16(scratch)) {
      return Fail(kInvalid, "%s: an f32 x needs %zu bytes of 16-byte aligned scratch for its bf16 copy, got %zu", op, need, scratch_bytes);
    }
    const size_t count = static_cast<size_t>(m) * k;
    e = LaunchToBf16(x, scratch, count, st);
    if (e != cudaSuccess) return CudaFail("INT8_PROJ_SWIGLU activation cast", e);
    CountLaunches(1);
    xb = reinterpret_cast<const __nv_bfloat16*>(scratch);
  }
  e = PrepareInt8GemmTcKernels();
  if (e != cudaSuccess) return CudaFail("INT8_PROJ_SWIGLU set-up", e);
  int launches = 0;
  e = LaunchInt8GemmTc(xb, codes, scales, nullptr, y, y_dtype, m, k, n, st, &launches, (flags & TLALOC_B200_GEMM_WEIGHTS_CONST) != 0, true);
  if (e != cudaSuccess) return CudaFail("INT8_PROJ_SWIGLU tensor-core launch", e);
  CountLaunches(launches);
  return kOk;
}
