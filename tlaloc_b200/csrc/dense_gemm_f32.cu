// The f32 projection on the tensor cores (include/tlaloc_b200.h, tlaloc_b200_dense_gemm): every f32 operand is the exact sum of three
// bf16 numbers (8 + 8 + 8 bits of its 24), and the six products of parts that reach f32's last place run as tcgen05.mma kind::f16.
//
// Accuracy.  Products of parts are exact; what is left out (middle x low, low x low) is below 2^-26 of a product and of either sign.  An
// accumulator in TMEM holds one chunk of 32 k only, its small products first and its large ones last; the chunks are summed in registers with
// rounding to nearest.  So a sum of k products has k / 32 rounded additions where the plain kernel (dense_gemm.cu) has k; but inside a chunk the
// tensor core cuts what it adds.  Error against 64 bits (2-norm over 200 x 512 sums, relative, 1e-7) and the plain kernel's:
//   k          4            16           32           128          2048         10304
//   normal     0.46  0.40   0.48  0.73   0.57  1.02   0.71  2.04   0.97  8.04   1.43  18.1
//   1 .. 1.001 0.69  0.43   0.69  0.63   0.69  0.81   0.78  1.51   0.82  5.91   0.84  15.7
// hence the plain kernel below k = 32.  A sum that one product outweighs is cut where the plain kernel rounds: 1.4e-7 and 0.3e-7 at worst (k = 32).
// bf16 ends where f32 does (2^-149 is f32's last place there, 2^-126 bf16's smallest normal number), so the parts of small operands would lose
// their low bits: operands are split after a multiplication by 2^24, which leaves every nonzero part normal, and a finished sum is
// multiplied by 2^-48.  What gets too large by that (an operand of 2^104, a sum of 2^80 and more), an infinity or a NaN makes a part infinite
// and the sum NaN or infinite: such an output is computed again with plain FMAs.
//
// D[n, m] = sum_k W[n, k] X[m, k]: 128 weight rows are the MMA's M, a tile of up to 208 activation rows its N.
//   producer lane boxes of 32 k of both operands by TMA (f32, 128-byte swizzle), two to eight stages ahead
//   sixteen warps split a chunk of 32 k into the three planes: the weights' go to TMEM (a lane a row; an MMA of 208 columns takes 114 cycles with A there, 148
//                 with A in shared memory, whose bandwidth the splits' stores need as well), the activations' to shared memory (128-byte swizzle; a
//                 buffer is one half of the planes' rows)
//   MMA lane      the six products of a chunk, into one of two accumulators
//   eight warps   add the finished accumulator to sums in registers (104 a thread at 208 rows, hence the register split), and write the tile
//   persistent    a CTA walks tiles;   K slices   the slices of a tile are a cluster and sum their partial tiles in rank order
// Bound at 208 rows by the split and the six products, which run side by side (203 rows, n 18944, k 2048: 106 us with the weights' planes in shared memory too, where
// each of the two alone took about 100; 92 us now, the split first: its warps wait for one another's latencies, with 40 registers there is one group of words at a time),
// at few rows by the way of a chunk through the three kinds of warps (0.8 us each).  203 rows, n 2048, k 10304: 77 us, 1414 us with plain FMAs; one
// row, n 32768, k 2048: 102 us, 443 us.  (72 registers a thread at launch: the 208-row form spills 92 bytes, the two smallest 16; none did with the planes in shared memory but the 64-row form, 8.)  Every mbarrier wait is bounded.  Sums computed again: 203 rows, n 18944, k 2048 with one row of NaN 0.26 ms, all
// infinite 2.2 ms (DenseGemmTiled 0.85 ms); n 2048, k 10304: 0.80, 2.3 (1.4) ms.
#include <cuda.h>

#include "common.cuh"
#include "dense_gemm.cuh"
#include "tc_common.cuh"

namespace tlaloc_b200 {
namespace {

using namespace tc;

constexpr int kBN = 128, kBK = 32, kSumWarps = 8, kSplitWarps = 16, kMmaWarp = kSumWarps + kSplitWarps, kProducerWarp = kMmaWarp + 1;
constexpr int kThreads = (kMmaWarp + 4) * 32;
constexpr int kOutUnits = 4;

// BT: most activation rows of a tile.
template <int BT>
struct Layout {
  static constexpr int kPlane = BT * 128;  // of the activations, 64 k a row: two buffers of 32
  static constexpr int kRaw = 3 * kPlane;
  static constexpr int kStage = (kBN + BT) * 128;
  static constexpr int kStages = BT == 208 ? 2 : BT == 128 ? 3 : BT == 64 ? 6 : 8;
  static constexpr int kTileStride = kBN + 4;  // a slice's partial tile [BT][kTileStride] f32, aliases the planes and the ring
  static constexpr int kOut = kRaw + kStages * kStage;  // what each sum warp has finished of its tile, kOutUnits of its units at a time
  static_assert(kOut >= BT * kTileStride * 4, "the partial tile aliases the planes and the ring");
  static constexpr int kBars = kOut + kSumWarps * kOutUnits * 8 * 32 * 4;
  static constexpr int kSlot = kBars + 8 * (6 + 2 * kStages);
  static constexpr int kBytes = kSlot + 16 + 1024;  // slack to align to 1024
  // Registers a thread of the three kinds of warpgroups; 128 * (2 * sum + 4 * split + mma) is the 896 * 72 of the launch.
  static constexpr int kSumRegs = 152, kSplitRegs = 40, kMmaRegs = 40;
  static_assert(128 * (2 * kSumRegs + 4 * kSplitRegs + kMmaRegs) <= kThreads * 72, "more registers than the launch has");
  static constexpr int kUnits = BT / 16;           // groups of eight activation rows a thread sums
  // TMEM: two accumulators kAcc columns apart, and the weights' three planes of a chunk, sixteen columns each, twice.
  static constexpr int kAcc = BT == 208 ? 224 : BT;
  static constexpr uint32_t kCols = BT >= 128 ? 512 : 256;
  __device__ static constexpr uint32_t PlaneColumn(int buffer, int plane)
  {
    const int i = buffer * 3 + plane;
    if (BT == 208) return i < 5 ? 432 + 16 * i : 208;  // the last one between the accumulators
    return 2 * kAcc + 16 * i;
  }
};

struct F32Args {
  tlaloc_b200_dense_problem p[2];
  int M[2], tiles_m[2], tiles_n[2];
  int swap_x[2];  // the activations' map has the batch before the rows
  int tiles0, tiles, ks, bt, weights_const, groups;  // groups: of the last problem, whose tiles are not counted here
};

__device__ int g_f32_status = 0;  // nonzero after an mbarrier wait timed out (sticky until read)

struct Tile {
  int pr, n0, m0, b, M;  // M: first row that is not the tile's to write
};
__device__ __forceinline__ Tile TileAt(const F32Args& a, int id, const int* start)
{
  Tile t;
  t.pr = id >= a.tiles0 ? 1 : 0;
  if (t.pr) id -= a.tiles0;
  const tlaloc_b200_dense_problem& p = a.p[t.pr];
  if (p.row_offsets != nullptr) {
    int lo = 0, hi = a.groups;  // start[lo] <= id < start[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (start[mid] <= id) lo = mid;
      else hi = mid;
    }
    id -= start[lo];
    t.b = lo;
    const int tiles_m = (start[lo + 1] - start[lo]) / a.tiles_n[t.pr];
    t.M = min(p.row_offsets[lo + 1], a.M[t.pr]);
    t.m0 = p.row_offsets[lo] + (id % tiles_m) * a.bt;
    t.n0 = (id / tiles_m) * kBN;
    return t;
  }
  t.M = a.M[t.pr];
  t.m0 = (id % a.tiles_m[t.pr]) * a.bt;  // activation tiles of one weight tile run side by side: the weights leave HBM once
  id /= a.tiles_m[t.pr];
  t.n0 = (id % a.tiles_n[t.pr]) * kBN;
  t.b = id / a.tiles_n[t.pr];
  return t;
}

// Two f32 times 2^24 as the exact sum of three pairs of bf16, each rounded to nearest from what the parts before it leave: after it the lowest
// bit of any f32 is 2^-125 or above, so no part is subnormal.
constexpr float kDown = 0x1p-48f;  // what a sum is multiplied by
__device__ __forceinline__ void Split2(uint64_t xy, uint32_t& h, uint32_t& m, uint32_t& l)
{
  // v's pair of bf16, and what it leaves of v
  auto part = [](uint64_t v, uint32_t& out) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    out = *reinterpret_cast<const uint32_t*>(&b);
    uint64_t there;
    asm("mov.b64 %0, {%1, %2};" : "=l"(there) : "r"(out << 16), "r"(out & 0xffff0000u));
    return there;
  };
  constexpr uint64_t kUp2 = 0x4b8000004b800000ull, kMinus2 = 0xbf800000bf800000ull;  // 2^24 and -1, twice
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(xy) : "l"(kUp2));
  uint64_t at = part(xy, h);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(xy) : "l"(at), "l"(kMinus2));
  at = part(xy, m);
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(xy) : "l"(at), "l"(kMinus2));
  part(xy, l);
}

__device__ __forceinline__ bool Doubtful(float v) { return !(fabsf(v) < INFINITY); }

__device__ __forceinline__ const float* XRow(const tlaloc_b200_dense_problem& p, const Tile& t, int m)
{
  return static_cast<const float*>(p.x) + (p.row_offsets != nullptr ? 0 : p.batch_x * t.b) + static_cast<size_t>(m) * p.ld_x;
}
__device__ __forceinline__ const float* WRow(const tlaloc_b200_dense_problem& p, const Tile& t, int n)
{
  return static_cast<const float*>(p.w) + p.batch_w * t.b + static_cast<size_t>(n) * p.k;
}
__device__ __forceinline__ void Put(const tlaloc_b200_dense_problem& p, size_t at, float v)
{
  if (p.y_dtype == TLALOC_B200_F32) static_cast<float*>(p.y)[at] = v;
  else static_cast<__nv_bfloat16*>(p.y)[at] = __float2bfloat16_rn(v);
}

// Eight sums again with plain FMAs in k order (the plain kernel's bits): rows 0 .. last of x, ld apart, with a column of w a lane, by the whole warp.
// Bound by the way of its words (the columns' are scattered); two steps' loads are in flight.  The rest of the CTA waits meanwhile, so it counts its
// progress at `beat` (MbarWaitAlive).
struct Sums {
  float v[8];
};
__device__ __noinline__ Sums PlainSums(const float* x, size_t ld, int last, const float* w, int K, volatile uint32_t* beat)
{
  Sums s = {};
#pragma unroll 2
  for (int k = 0; k < K; k += 4) {
    const float4 b = *reinterpret_cast<const float4*>(w + k);
    float4 a[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = *reinterpret_cast<const float4*>(x + min(c, last) * ld + k);
#pragma unroll
    for (int c = 0; c < 8; ++c) s.v[c] = fmaf(a[c].w, b.w, fmaf(a[c].z, b.z, fmaf(a[c].y, b.y, fmaf(a[c].x, b.x, s.v[c]))));
    if ((k & 511) == 0 && (threadIdx.x & 31) == 0) atomicAdd(const_cast<uint32_t*>(beat), 1u);
  }
  return s;
}

// MbarWait that goes on while `words[1]` counts: sums that are computed again may take longer than the limit.
__device__ __forceinline__ bool MbarWaitOn(uint32_t bar, uint32_t parity, volatile uint32_t* words)
{
  for (;;) {
    const uint32_t seen = words[1];
    if (MbarPoll(bar, parity, words)) return true;
    if (words[0] != 0u || words[1] == seen) break;
  }
  words[0] = 1u;
  return false;
}
__device__ __forceinline__ bool MbarWaitAlive(uint32_t bar, uint32_t parity, volatile uint32_t* words)
{
  return MbarPoll(bar, parity, words) || MbarWaitOn(bar, parity, words);
}
__device__ __forceinline__ bool MbarWaitAliveWarp(uint32_t bar, uint32_t parity, int lane, volatile uint32_t* words)
{
  int ok = 1;
  if (lane == 0) ok = MbarWaitAlive(bar, parity, words) ? 1 : 0;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

// A tile is finished in two passes: what is sure is stored at once, the rest is computed again when the sums in registers are gone and only
// bits say which; doing both at once cost registers on the way of every tile (203 rows, n 18944, k 2048: 118 us, 109 so).
// Which of a lane's eight sums (times 2^48) have to be computed again, as bits; of a gated pair both have.
__device__ __forceinline__ uint32_t DoubtfulBits(const tlaloc_b200_dense_problem& p, int n, int m, int step, int end, const float* v)
{
  uint32_t bits = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) bits |= m + c * step < end && Doubtful(v[c]) ? 1u << c : 0u;
  if (n >= p.n) bits = 0;
  return IsGated(p.act) ? bits | __shfl_xor_sync(0xffffffffu, bits, kGateBlock) : bits;
}

// Eight finished sums of column n (a warp's lanes hold 32 consecutive columns), rows m, m + step, ... below end: epilogue and store of those whose bit is set.
__device__ __forceinline__ void Finish(const tlaloc_b200_dense_problem& p, const Tile& t, int n, int m, int step, int end, const float* v, uint32_t bits)
{
  constexpr int kU = 8;
  const size_t out = p.row_offsets != nullptr ? 0 : p.batch_y * t.b;
  if (IsGated(p.act)) {  // gate and other factor are sixteen lanes apart
#pragma unroll
    for (int c = 0; c < kU; ++c) {
      const int r = m + c * step;
      const float other = __shfl_xor_sync(0xffffffffu, v[c], kGateBlock);
      if (n < p.n && r < end && (n & kGateBlock) == 0 && (bits >> c & 1u) != 0) {
        Put(p, out + static_cast<size_t>(r) * p.ld_y + (n >> 5) * kGateBlock + (n & 15), GatedValue(p.act, v[c], other));
      }
    }
    return;
  }
  if (n >= p.n) return;
  // What is the same for all eight is asked once, ahead of them: few warps are left here, and a chain of questions for each value was most of a short tile's
  // time.
  const int64_t y_step = step * p.ld_y;
  const size_t at = out + static_cast<size_t>(m) * p.ld_y + n;
  float o[kU];
  const float bias = p.bias != nullptr ? __ldg(p.bias + n) : 0.f;
#pragma unroll
  for (int c = 0; c < kU; ++c) {
    o[c] = v[c] + bias;
    if (m + c * step >= end) bits &= ~(1u << c);
  }
  if (p.act != TLALOC_B200_ACT_NONE) {
#pragma unroll
    for (int c = 0; c < kU; ++c) o[c] = DenseActivation(p.act, o[c]);
  }
  if (p.residual != nullptr) {
    const float* from = p.residual + static_cast<size_t>(m) * p.ld_res + n;
    const int64_t r_step = step * p.ld_res;
    float res[kU];
#pragma unroll
    for (int c = 0; c < kU; ++c) res[c] = (bits >> c & 1u) != 0 ? from[c * r_step] : 0.f;
#pragma unroll
    for (int c = 0; c < kU; ++c) o[c] += res[c];
  }
  if (p.y_dtype == TLALOC_B200_F32) {
    float* y = static_cast<float*>(p.y) + at;
#pragma unroll
    for (int c = 0; c < kU; ++c)
      if ((bits >> c & 1u) != 0) y[c * y_step] = o[c];
  } else {
    __nv_bfloat16* y = static_cast<__nv_bfloat16*>(p.y) + at;
#pragma unroll
    for (int c = 0; c < kU; ++c)
      if ((bits >> c & 1u) != 0) y[c * y_step] = __float2bfloat16_rn(o[c]);
  }
}

// The same for sums still times 2^48; leaves the bits of those that are not stored.
__device__ __forceinline__ uint32_t FinishSure(const tlaloc_b200_dense_problem& p, const Tile& t, int n, int m, int step, int end, float* v)
{
  const uint32_t doubt = DoubtfulBits(p, n, m, step, end, v);
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] *= kDown;
  Finish(p, t, n, m, step, end, v, ~doubt);
  return doubt;
}
__device__ __forceinline__ void FinishDoubtful(const tlaloc_b200_dense_problem& p, const Tile& t, int n, int m, int step, int end, uint32_t bits,
                                               volatile uint32_t* beat)
{
  if (!__any_sync(0xffffffffu, bits != 0)) return;
  const Sums s = PlainSums(XRow(p, t, m), static_cast<size_t>(step) * p.ld_x, (end - 1 - m) / step, WRow(p, t, min(n, p.n - 1)), p.k, beat);
  Finish(p, t, n, m, step, end, s.v, bits);
}

__device__ __forceinline__ void ClusterSync()
{
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void TcLd8(uint32_t taddr, uint32_t* r)
{
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void TcSt4(uint32_t taddr, const uint32_t (&r)[4])
{
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%4], {%0, %1, %2, %3};\n" ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(taddr) : "memory");
}

// The chunks of a tile that a CTA sums: all of them, or the slice of its cluster rank.
__device__ __forceinline__ int Chunks(const F32Args& a, const Tile& t, int& first)
{
  const int nb = (a.p[t.pr].k + kBK - 1) / kBK;
  if (a.ks <= 1) {
    first = 0;
    return nb;
  }
  const int per = (nb + a.ks - 1) / a.ks;
  first = static_cast<int>(blockIdx.y) * per;
  return max(0, min(per, nb - first));
}

// x (the k coordinate) is a multiple of 32 f32: always a 16-byte boundary.
__device__ __forceinline__ void TmaBox3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar, uint64_t policy)
{
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;\n" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(bar), "l"(policy)
      : "memory");
}

template <int BT>
__global__ void __launch_bounds__(kThreads, 1)
    DenseGemmF32Kernel(const __grid_constant__ CUtensorMap w0, const __grid_constant__ CUtensorMap x0, const __grid_constant__ CUtensorMap w1,
                       const __grid_constant__ CUtensorMap x1, const __grid_constant__ F32Args a)
{
  using L = Layout<BT>;
  constexpr int S = L::kStages;
  constexpr uint32_t kCols = L::kCols;
  extern __shared__ unsigned char smem_raw[];
  __shared__ int s_start[kMaxGroups + 1];
  const uint32_t base = (SmemAddr(smem_raw) + 1023u) & ~1023u;  // the swizzle is a function of address bits 4..9
  unsigned char* smem = smem_raw + (base - SmemAddr(smem_raw));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t full = base + L::kBars, done = full + 16, empty = done + 16;  // planes written; a chunk's MMAs through; its accumulator added
  const uint32_t landed = empty + 16, freed = landed + 8 * S;                                      // a stage's boxes are there; split
  volatile uint32_t* slot = reinterpret_cast<volatile uint32_t*>(smem + L::kSlot);
  volatile uint32_t* words = slot + 1;  // abort word; progress of sums computed again
  if (tid == 0) {
    words[0] = words[1] = 0u;
    for (int i = 0; i < 2; ++i) {
      MbarInit(full + 8 * i, kSplitWarps);
      MbarInit(done + 8 * i, 1);
      MbarInit(empty + 8 * i, kSumWarps);
    }
    for (int i = 0; i < S; ++i) {
      MbarInit(landed + 8 * i, 1);
      MbarInit(freed + 8 * i, kSplitWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(base + L::kSlot), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *slot;
  const bool early = a.weights_const != 0 && a.groups == 0;  // the first weights travel before the dependency wait
  if (!early || warp != kProducerWarp) GridDependencySync();
  int tiles = a.tiles;
  if (a.groups > 0) {
    const int pr = a.p[1].row_offsets != nullptr ? 1 : 0;
    const int* offsets = a.p[pr].row_offsets;
    if (warp == 0) {
      int total = 0;
      for (int e0 = 0; e0 < a.groups; e0 += 32) {
        const int e = e0 + lane;
        int v = e < a.groups ? max(0, (min(offsets[e + 1], a.M[pr]) - offsets[e] + a.bt - 1) / a.bt) * a.tiles_n[pr] : 0;
        const int own = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= o) v += u;
        }
        if (e < a.groups) s_start[e] = total + v - own;
        total += __shfl_sync(0xffffffffu, v, 31);
      }
      if (lane == 0) s_start[a.groups] = total;
    }
    __syncthreads();
    tiles += s_start[a.groups];
  }
  bool ok = true;
  int it = 0;  // chunks so far: chunk `it` has buffer and accumulator it & 1

  if (warp >= kMmaWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(L::kMmaRegs));
    if (warp == kMmaWarp && ElectOne()) {
      // f32 accumulator, bf16 A and B, both K-major, M = 128
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a.bt >> 3) << 17) | (8u << 24);
      const uint64_t xd = SmemDesc(base, 16, 1024);
      for (int id = blockIdx.x; id < tiles; id += gridDim.x) {
        const Tile t = TileAt(a, id, s_start);
        int first;
        const int nb = Chunks(a, t, first);
        for (int c = 0; c < nb; ++c, ++it) {
          const int b = it & 1;
          if (it >= 2) ok = MbarWaitAlive(empty + 8 * b, ((it >> 1) - 1) & 1, words) && ok;
          ok = MbarWaitAlive(full + 8 * b, (it >> 1) & 1, words) && ok;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint32_t acc = tmem + b * L::kAcc;
          constexpr uint32_t P = L::kPlane >> 4;
          const uint64_t x = xd + 4 * b;
          const uint32_t high = tmem + L::PlaneColumn(b, 0), middle = tmem + L::PlaneColumn(b, 1), low = tmem + L::PlaneColumn(b, 2);
          // planes high, middle, low: small products first
          TcMmaTmemA(acc, high, x + 2 * P, idesc, 0u);
          TcMmaTmemA(acc, high + 8, x + 2 * P + 2, idesc, 1u);
          TcMmaTmemA(acc, low, x, idesc, 1u);
          TcMmaTmemA(acc, low + 8, x + 2, idesc, 1u);
          TcMmaTmemA(acc, middle, x + P, idesc, 1u);
          TcMmaTmemA(acc, middle + 8, x + P + 2, idesc, 1u);
          TcMmaTmemA(acc, high, x + P, idesc, 1u);
          TcMmaTmemA(acc, high + 8, x + P + 2, idesc, 1u);
          TcMmaTmemA(acc, middle, x, idesc, 1u);
          TcMmaTmemA(acc, middle + 8, x + 2, idesc, 1u);
          TcMmaTmemA(acc, high, x, idesc, 1u);
          TcMmaTmemA(acc, high + 8, x + 2, idesc, 1u);
          TcCommit(done + 8 * b);
        }
      }
      if (!ok) atomicExch(&g_f32_status, 1);
    } else if (warp == kProducerWarp && ElectOne()) {
      uint64_t w_policy, x_policy;
      if (a.tiles_m[0] == 1) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(w_policy));
      else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;\n" : "=l"(w_policy));
      asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(x_policy));
      const uint32_t bytes = (kBN + a.bt) * 128;
      int s = 0, round = 0;  // the next stage, and how often the ring has been around
      bool waited = !early;
      for (int id = blockIdx.x; id < tiles; id += gridDim.x) {
        const Tile t = TileAt(a, id, s_start);
        int first;
        const int nb = Chunks(a, t, first);
        auto load_x = [&](int c, int at) {
          const int z = a.p[t.pr].row_offsets != nullptr ? 0 : t.b;
          const bool swap = a.swap_x[t.pr] != 0;
          TmaBox3d(base + L::kRaw + at * L::kStage + kBN * 128, t.pr ? &x1 : &x0, (first + c) * kBK, swap ? z : t.m0, swap ? t.m0 : z, landed + 8 * at, x_policy);
        };
        auto load_w = [&](int c, int at) {
          MbarExpectTx(landed + 8 * at, bytes);
          TmaBox3d(base + L::kRaw + at * L::kStage, t.pr ? &w1 : &w0, (first + c) * kBK, t.n0, t.b, landed + 8 * at, w_policy);
        };
        int c = 0;
        if (!waited) {  // constant weights of the first stages travel before the dependency wait; activations only after it
          const int ahead = min(nb, S);
          for (int i = 0; i < ahead; ++i) load_w(i, i);
          GridDependencySync();
          waited = true;
          for (; c < ahead; ++c) load_x(c, c);
          s = ahead == S ? 0 : ahead;
          round = ahead == S ? 1 : 0;
        }
        for (; c < nb; ++c) {
          if (round > 0) ok = MbarWaitAlive(freed + 8 * s, (round - 1) & 1, words) && ok;
          load_w(c, s);
          load_x(c, s);
          if (++s == S) {
            s = 0;
            ++round;
          }
        }
      }
      if (!waited) GridDependencySync();
      if (!ok) {  // given up: let the copies in flight land before the CTA's shared memory goes away
        atomicExch(&g_f32_status, 1);
        volatile uint32_t never = 0;
        for (int i = 0; i < S; ++i) {
          const int uses = round + (i < s ? 1 : 0);
          if (uses > 0) MbarWait(landed + 8 * i, (uses - 1) & 1, &never);
        }
      }
    }
    __syncwarp();
    if (a.ks > 1) {
      ClusterSync();
      ClusterSync();
    }
  } else if (warp >= kSumWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(L::kSplitRegs));
    // Weights: a thread has a row of the warp's TMEM lanes and eight k, two 16-byte words of a row of the stage (the eight lanes of a phase have them in
    // different places by the swizzle) and four columns of each plane.
    // Activations: a lane's eight k are two words of a row of the stage and one of each plane's; four lanes a row, and the two rows of a phase of
    // eight lanes differ by 5 in their swizzle, so that neither the loads (words 0 2 4 6 of a row) nor the stores (words 0 - 3, or 4 - 7) collide.
    const int sw = warp - kSumWarps, u = lane & 3, low = (lane >> 3) ^ ((lane & 4) != 0 ? 5 : 0), w_row = (warp & 3) * 32 + lane, w_k = sw >> 2;
    const uint32_t w_from = base + L::kRaw + w_row * 128 + (((2 * w_k) ^ (w_row & 7)) << 4);
    const uint32_t w_to = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 4 * w_k;
    const uint32_t from0 = base + L::kRaw + kBN * 128 + low * 128 + (((2 * u) ^ low) << 4), to0 = base + low * 128 + ((u ^ low) << 4);
    const int groups = a.bt >> 3;  // of eight rows of activations
    int s = 0, phase = 0;
    for (int id = blockIdx.x; id < tiles; id += gridDim.x) {
      const Tile t = TileAt(a, id, s_start);
      int first;
      const int nb = Chunks(a, t, first);
      for (int c = 0; c < nb; ++c, ++it) {
        ok = MbarWaitAliveWarp(landed + 8 * s, phase, lane, words) && ok;
        if (it >= 2) ok = MbarWaitAliveWarp(done + 8 * (it & 1), ((it >> 1) - 1) & 1, lane, words) && ok;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t from = from0 + s * L::kStage, to = to0 ^ ((it & 1) << 6);
        auto split = [](uint32_t at, uint32_t (&part)[3][4]) {
          uint64_t v[4];
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];\n" : "=l"(v[0]), "=l"(v[1]) : "r"(at));
          asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];\n" : "=l"(v[2]), "=l"(v[3]) : "r"(at ^ 16));
#pragma unroll
          for (int e = 0; e < 4; ++e) Split2(v[e], part[0][e], part[1][e], part[2][e]);
        };
        {
          uint32_t part[3][4];
          split(w_from + s * L::kStage, part);
#pragma unroll
          for (int q = 0; q < 3; ++q) TcSt4(w_to + ((it & 1) != 0 ? L::PlaneColumn(1, q) : L::PlaneColumn(0, q)), part[q]);
        }
        if constexpr (BT <= 64) {
          // Few rows: half a group a warp, so that all sixteen have some (64 rows, n 32768, k 2048: 127.6 us with whole groups for half of the warps, 124.4 so; one row 105.7, 102.3). A
          // lane has four k, and the two rows of sixteen lanes lie in different halves of their lines.
          const int row = (sw >> 1) * 8 + 2 * (sw & 1) + ((lane & 8) >> 1) + (lane >> 4), word = lane & 7;
          if ((sw >> 1) < groups) {
            uint64_t v[2];
            uint32_t part[3][2];
            asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];\n" : "=l"(v[0]), "=l"(v[1]) : "r"(base + L::kRaw + s * L::kStage + (kBN + row) * 128 + ((word ^ (row & 7)) << 4)));
#pragma unroll
            for (int e = 0; e < 2; ++e) Split2(v[e], part[0][e], part[1][e], part[2][e]);
            const uint32_t at = (base + row * 128 + (((word >> 1) ^ (row & 7)) << 4) + (word & 1) * 8) ^ ((it & 1) << 6);
#pragma unroll
            for (int q = 0; q < 3; ++q) asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at + q * L::kPlane), "r"(part[q][0]), "r"(part[q][1]) : "memory");
          }
        } else {
#pragma unroll
          for (int i = 0; i < BT / 8; i += kSplitWarps) {
            const int g = i + sw;
            if (g >= groups) break;
            uint32_t part[3][4];
            split(from + g * 1024, part);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(to + g * 1024 + q * L::kPlane), "r"(part[q][0]), "r"(part[q][1]),
                           "r"(part[q][2]), "r"(part[q][3])
                           : "memory");
            }
          }
        }
        asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          MbarArrive(full + 8 * (it & 1));
          MbarArrive(freed + 8 * s);
        }
        if (++s == S) {
          s = 0;
          phase ^= 1;
        }
      }
    }
    if (!ok) atomicExch(&g_f32_status, 1);
    if (a.ks > 1) {
      ClusterSync();
      ClusterSync();
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(L::kSumRegs));
    const int quad = warp & 3, col0 = (warp >> 2) * (a.bt >> 1), units = a.bt >> 4;  // this warp's lanes and columns of an accumulator
    for (int id = blockIdx.x; id < tiles; id += gridDim.x) {
      const Tile t = TileAt(a, id, s_start);
      const tlaloc_b200_dense_problem& p = a.p[t.pr];
      int first;
      const int nb = Chunks(a, t, first);
      float acc[L::kUnits][8];
#pragma unroll
      for (int q = 0; q < L::kUnits; ++q)
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[q][e] = 0.f;
      for (int c = 0; c < nb; ++c, ++it) {
        ok = MbarWaitAliveWarp(done + 8 * (it & 1), (it >> 1) & 1, lane, words) && ok;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t from = tmem + (static_cast<uint32_t>(quad * 32) << 16) + (it & 1) * L::kAcc + col0;
#pragma unroll
        for (int q = 0; q < L::kUnits; q += 2) {
          if (q < units) {
            uint32_t r[2][8];
            TcLd8(from + q * 8, r[0]);
            if (q + 1 < L::kUnits) TcLd8(from + q * 8 + 8, r[1]);  // within the accumulator's columns also where the tile ends before it
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              acc[q][e] += __uint_as_float(r[0][e]);
              if (q + 1 < L::kUnits) acc[q + 1 < L::kUnits ? q + 1 : q][e] += __uint_as_float(r[1][e]);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) MbarArrive(empty + 8 * (it & 1));
      }
      if (a.ks <= 1) {
        // Through shared memory, a few units at a time, so that there is one copy of the epilogue's code: unrolled over the registers it was 470 KB, all
        // of which a tile fetched once (203 rows, n 128, k 32: 26.1 us, 22.2 so, 14.4 with the epilogue's questions asked once for eight values).
        const int n = t.n0 + quad * 32 + lane, m = t.m0 + col0;
        constexpr int kRounds = (L::kUnits + kOutUnits - 1) / kOutUnits;
        float* place = reinterpret_cast<float*>(smem + L::kOut) + warp * (kOutUnits * 8 * 32) + lane;
        uint32_t doubt[kRounds] = {};
#pragma unroll 1
        for (int i = 0; i < kRounds; ++i) {
          __syncwarp();
#pragma unroll
          for (int q = 0; q < L::kUnits; ++q) {
            if (q / kOutUnits == i) {
#pragma unroll
              for (int e = 0; e < 8; ++e) place[((q % kOutUnits) * 8 + e) * 32] = acc[q][e];
            }
          }
          __syncwarp();
          uint32_t bits = 0;
#pragma unroll 1
          for (int q = i * kOutUnits; q < min(units, (i + 1) * kOutUnits); ++q) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = place[((q % kOutUnits) * 8 + e) * 32];
            bits |= FinishSure(p, t, n, m + q * 8, 1, t.M, v) << 8 * (q % kOutUnits);
          }
#pragma unroll
          for (int j = 0; j < kRounds; ++j) doubt[j] = j == i ? bits : doubt[j];
        }
#pragma unroll 1
        for (int i = 0; i < kRounds; ++i) {
          uint32_t bits = 0;
#pragma unroll
          for (int j = 0; j < kRounds; ++j) bits = j == i ? doubt[j] : bits;
#pragma unroll 1
          for (int q = 0; q < kOutUnits && __any_sync(0xffffffffu, bits != 0); ++q, bits >>= 8) {
            FinishDoubtful(p, t, n, m + (i * kOutUnits + q) * 8, 1, t.M, bits & 255u, words + 1);
          }
        }
      } else {
        float* tile = reinterpret_cast<float*>(smem);  // over the planes and the ring: every chunk of this CTA's one tile has been split, every MMA is through
#pragma unroll
        for (int q = 0; q < L::kUnits; ++q) {
          if (q < units) {
#pragma unroll
            for (int e = 0; e < 8; ++e) tile[(col0 + q * 8 + e) * L::kTileStride + quad * 32 + lane] = acc[q][e];
          }
        }
      }
    }
    if (!ok) atomicExch(&g_f32_status, 1);
    if (a.ks > 1) {
      ClusterSync();  // every slice's tile is in its CTA's shared memory
      cg::cluster_group cluster = cg::this_cluster();
      const Tile t = TileAt(a, blockIdx.x, s_start);
      const tlaloc_b200_dense_problem& p = a.p[t.pr];
      const int nl = tid & 127, nr = static_cast<int>(cluster.num_blocks()), rows = min(a.bt, t.M - t.m0), step = 2 * nr;
      float* tile = reinterpret_cast<float*>(smem);
      constexpr int kU = 8;
      for (int c0 = static_cast<int>(cluster.block_rank()) + nr * (tid >> 7); c0 < rows; c0 += kU * step) {
        float v[kU] = {};
        for (int q = 0; q < nr; ++q) {
          const float* peer = cluster.map_shared_rank(tile, q) + nl;
          float w[kU];
#pragma unroll
          for (int e = 0; e < kU; ++e) w[e] = c0 + e * step < rows ? peer[(c0 + e * step) * L::kTileStride] : 0.f;
#pragma unroll
          for (int e = 0; e < kU; ++e) v[e] += w[e];
        }
        const uint32_t doubt = FinishSure(p, t, t.n0 + nl, t.m0 + c0, step, t.m0 + rows, v);
        FinishDoubtful(p, t, t.n0 + nl, t.m0 + c0, step, t.m0 + rows, doubt, words + 1);
      }
      ClusterSync();  // no CTA leaves while a peer may still read its tile
    }
    asm volatile("bar.sync 1, 256;\n" ::: "memory");
    if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
    }
  }
}

// ---- host -----------------------------------------------------------------------------------------------------------

int g_slots[kMaxDevices][9];  // resident CTAs when launched as clusters of ks: measured for one layout, every one of which fills an SM's shared memory

cudaError_t PrepareDenseF32()
{
  static OncePerDevice once;
  return once.Run([](int device) {
    TensorMapEncoder();
    cudaError_t e = cudaSuccess;
#define TLALOC_OPT_IN(BT) \
  if (e == cudaSuccess) e = cudaFuncSetAttribute(DenseGemmF32Kernel<BT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Layout<BT>::kBytes)
    TLALOC_OPT_IN(32);
    TLALOC_OPT_IN(64);
    TLALOC_OPT_IN(128);
    TLALOC_OPT_IN(208);
#undef TLALOC_OPT_IN
    if (e != cudaSuccess) return e;
    for (int ks = 1; ks <= 8; ++ks) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(148, ks, 1);
      cfg.blockDim = dim3(kThreads, 1, 1);
      cfg.dynamicSmemBytes = Layout<128>::kBytes;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1;
      attr[0].val.clusterDim.y = ks;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int clusters = 0;
      if (cudaOccupancyMaxActiveClusters(&clusters, DenseGemmF32Kernel<128>, &cfg) != cudaSuccess || clusters <= 0) {
        cudaGetLastError();
        clusters = (ks <= 2 ? 148 : ks <= 4 ? 128 : 112) / ks;
      }
      g_slots[device][ks] = clusters * ks;
    }
    return cudaSuccess;
  });
}

int ReadF32Status()
{
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_f32_status, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_f32_status, &zero, sizeof(int));
  }
  return v;
}
KernelSetup g_setup(PrepareDenseF32, ReadF32Status);

// K slices (1..8) of tiles with k of nb times 64, in microseconds: 64 k took 3.6 us at 208 rows and 1.7 us at
// few with all planes in shared memory, which is what the counts were fitted to (2.9 and 1.6 since the weights' are in TMEM); a tile's start and end cost about 3 us, a cluster's sum 2 us and more with its ranks.
int ChooseSlices(long long tiles, int nb, int bt)
{
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= kMaxDevices) device = 0;
  const double chunk = fmax(1.7, 3.6 * bt / 208);
  int best = 1;
  double best_cost = 1e30;
  for (int ks = 1; ks <= 8; ++ks) {
    if (ks > 1 && nb / ks < 2) break;
    const int slots = g_slots[device][ks] > 0 ? g_slots[device][ks] : 148 / ks * ks;
    const long long waves = (tiles * ks + slots - 1) / slots;
    const double cost = waves * ((nb + ks - 1) / ks * chunk + 3.0 + (ks > 1 ? 1.5 + 0.2 * ks : 0.0));
    if (cost < best_cost * 0.97) {
      best_cost = cost;
      best = ks;
    }
  }
  return best;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// f32 [batch][rows][k] with strides in elements, boxes of 32 k x box_rows rows; the dimension with the smaller stride comes first (*swap: the batch).
bool EncodeMatrix(CUtensorMap* map, const void* ptr, int64_t k, int64_t rows, int64_t batch, int64_t ld, int64_t batch_stride, uint32_t box_rows, int* swap)
{
  auto encode = reinterpret_cast<EncodeTiledFn>(TensorMapEncoder());
  if (encode == nullptr) return false;
  *swap = batch > 1 && batch_stride < ld ? 1 : 0;
  if (batch == 1) batch_stride = ld;
  const cuuint64_t r_dim = static_cast<cuuint64_t>(rows), b_dim = static_cast<cuuint64_t>(batch);
  const cuuint64_t r_str = static_cast<cuuint64_t>(ld) * 4, b_str = static_cast<cuuint64_t>(batch_stride) * 4;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(k), *swap ? b_dim : r_dim, *swap ? r_dim : b_dim};
  const cuuint64_t strides[2] = {*swap ? b_str : r_str, *swap ? r_str : b_str};
  const cuuint32_t box[3] = {kBK, *swap ? 1u : box_rows, *swap ? box_rows : 1u};
  const cuuint32_t elem[3] = {1, 1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(ptr), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BT>
cudaError_t Launch(const CUtensorMap* maps, const F32Args& a, int ctas, cudaStream_t st)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, a.ks, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = Layout<BT>::kBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  cfg.numAttrs = ChainAttributes(attr, a.ks > 1 ? a.ks : 0);
  cfg.attrs = attr;
  return cudaLaunchKernelEx(&cfg, DenseGemmF32Kernel<BT>, maps[0], maps[1], maps[2], maps[3], a);
}

}  // namespace

bool DenseGemmF32Applies(const tlaloc_b200_dense_problem& p, int m)
{
  const long long rows = p.rows > 0 ? p.rows : m;
  return p.k >= kBK && p.k % 4 == 0 && p.ld_x % 4 == 0 && Aligned16(p.x) && Aligned16(p.w) && (p.batch == 1 || (p.batch_x % 4 == 0 && p.batch_w % 4 == 0)) &&
         (p.batch == 1 || ((p.row_offsets != nullptr || p.batch_x >= p.k) && p.batch_w >= p.k)) && TensorMapEncoder() != nullptr &&
         (rows / 16 + p.batch + 1) * ((p.n + kBN - 1) / kBN) * (p.row_offsets != nullptr ? 1 : p.batch) < (1ll << 30);
}

cudaError_t LaunchDenseGemmF32(const tlaloc_b200_dense_problem* problems, int count, int m, bool weights_const, cudaStream_t st, bool* taken)
{
  *taken = true;
  cudaError_t e = PrepareDenseF32();
  if (e != cudaSuccess) return e;
  // Rows of a tile: what the problem has in equal parts of up to 208, or what a group has on average (one that has more takes several tiles).
  int typical = 1, nb = 1 << 30;
  for (int i = 0; i < count; ++i) {
    const int rows = problems[i].rows > 0 ? problems[i].rows : m;
    typical = max(typical, problems[i].row_offsets != nullptr ? (rows + problems[i].batch - 1) / problems[i].batch : rows);
    nb = min(nb, (problems[i].k + 63) / 64);
  }
  const int parts = (typical + 207) / 208;
  CUtensorMap maps[4];
  F32Args a = {};
  a.bt = ((typical + parts - 1) / parts + 15) / 16 * 16;
  a.weights_const = weights_const ? 1 : 0;
  for (int i = 0; i < count; ++i) {
    const tlaloc_b200_dense_problem& s = problems[i];
    a.p[i] = s;
    a.M[i] = s.rows > 0 ? s.rows : m;
    int swap_w = 0;
    if (!EncodeMatrix(&maps[2 * i], s.w, s.k, s.n, s.batch, s.k, s.batch_w, kBN, &swap_w) || swap_w ||
        !EncodeMatrix(&maps[2 * i + 1], s.x, s.k, a.M[i], s.row_offsets != nullptr ? 1 : s.batch, s.ld_x, s.batch_x, a.bt, &a.swap_x[i])) {
      *taken = false;  // strides that no tensor map has (2^40 bytes and more)
      return cudaSuccess;
    }
    a.tiles_m[i] = (a.M[i] + a.bt - 1) / a.bt;
    a.tiles_n[i] = (s.n + kBN - 1) / kBN;
    if (s.row_offsets != nullptr) a.groups = s.batch;
    else a.tiles += a.tiles_n[i] * a.tiles_m[i] * s.batch;
    if (i == 0) a.tiles0 = s.row_offsets != nullptr ? 1 << 30 : a.tiles;
  }
  if (count == 1) {
    maps[2] = maps[0];
    maps[3] = maps[1];
  }
  a.ks = a.groups > 0 ? 1 : ChooseSlices(a.tiles, nb, a.bt);
  const int ctas = a.groups > 0 ? 148 : a.ks > 1 ? a.tiles : min(a.tiles, 148);
  if (a.bt <= 32) return Launch<32>(maps, a, ctas, st);
  if (a.bt <= 64) return Launch<64>(maps, a, ctas, st);
  if (a.bt <= 128) return Launch<128>(maps, a, ctas, st);
  return Launch<208>(maps, a, ctas, st);
}

}  // namespace tlaloc_b200
