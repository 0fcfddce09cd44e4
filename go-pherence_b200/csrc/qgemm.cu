// Quantised weights times several activation rows on the 5th-generation tensor cores: f16 operands,
// f32 accumulators in TMEM, one kernel for every weight format and both device layouts.
//
// Stands behind nvidia.GemmMLX (backends/nvidia/runtime/mlx.go:395-431), GPUGGUFMatrix.
// ProjectBatchToBuffer (runtime/gguf_matrix.go:121-135) and GemmFP8E4M3Buffer (runtime/fp8.go:271-320)
// for prefill chunks and verifier batches.
//
// Arithmetic
//   * A operand (weights, the 128 rows of a tile), written to TMEM as f16 by converter warps, exact:
//       MLX4F  scale * (nibble - 8) * 2^10, at most 11 significant bits: weights whose scales allow it
//              (goph_mlx_weight::foldable; every checkpoint seen does), so thousands of elements accumulate in
//              one block of columns and nothing is scaled on the way out.
//       MLX4   the others: nibble n as the f16 subnormal n * 2^-24 (the masked nibble IS the bit pattern; the
//              nibbles at bits 4..7 of a half read as 16 n and meet activations scaled by 1/16), a block of
//              columns per 64 elements.
//       Q4_K   the nibble as a subnormal times the sub-block's 6-bit scale: sc * n has at most 10 bits (Q5_K:
//       Q5_K   11, the most an f16 holds), so a block of columns lasts a super-block.
//       Q6_K   q - 32, a block per 16 elements (an 8-bit scale times 6 bits does not fit).
//       Q8_0   the signed byte, a block per 32 elements.
//       FP8    e4m3 -> f16 (exact, NaN codes stay NaN), a block of 4096 elements (128 columns: of an item, at most 8192).
//   * B operand (activations): every row is scaled by a power of two so that its largest magnitude
//     lies in [2^14, 2^15), and written as the sum of up to three f16 values, each the rounding of
//     what the ones before it left over.  Three hold an f32 exactly down to 2^-39 of the row's largest
//     element (f32 sums do not see below that, unless the weights at the larger elements are zero); a bf16 needs
//     one.  A row with an infinity is scaled by 2^-113.  All pieces accumulate into the
//     same columns.  The preparation kernel notes per row and 256 elements how many pieces are not
//     zero: f32 buffers that hold bf16 values cost one pass of the tensor cores, not three.
//   * The affine term (biases or minima times the groups' sums of x) is one or two more K16 steps per
//     chunk in bf16: A the biases, B the sums in three bf16 pieces (exact).
//   * Epilogue: tcgen05.ld per block, times the block's scale, running sums in registers, f32.
//
// What bounds it: the hand-overs between the roles (a wait that succeeds at once costs a warp about a
// hundred cycles), the conversion, and in front of it all the preparation launch.  An MMA of M128 x N x
// K16 takes N/2 cycles with A in TMEM (measured down to N = 16; with A in shared memory 32 + N/4 below
// N = 128), so 256 elements of a tile and 64 columns take 512 cycles per piece.  The B tiles cross from
// the L2 once per row tile, which at 64 columns is more than an SM gets: with TT = 2 the two tiles of an
// item share each B tile.
//
// Work: items (group of TT row tiles, block of up to 64 or 128 activation rows).  The items of the last,
// partial wave are cut along K over the CTAs of a thread-block cluster, whose sums meet in shared memory,
// added in split order.
//
// A CTA, one per SM, 28 warps: W loader (tiled layouts: a bulk copy per 256 elements and tile, stored
// contiguously; row-major and streaming layouts: tiled TMA copies into the same image, rows and elements
// past the matrix zero-filled, see load_rows), B loader (a slot per half chunk, all of its pieces), 2 MMA warps, 16
// converter and 8 epilogue warps, half of them in either of two pipes (see the kernel).
// Every wait is bounded (~2 s); a waiter that gives up records a code (800+) and the CTA winds down.
//
// Measured (B200, a call among others, us; before: integer products of 4 or 8 rows, or the bf16 kernel's
// passes of 16 f32 or 64 bf16 rows):
//   Q8_0 4096x4096 x19 44.5 -> 15.1; Q4_K 14336x4096 x64 381 -> 29.3; MLX4 6144x4096 x100 f32 129 -> 20.7;
//   MLX4 8192x8192 x64 bf16 33.2 -> 21.8; FP8 28672x8192 x256 bf16 226 -> 103 to 123 by the box
#include <string.h>

#include <mutex>
#include <type_traits>

#include "qgemm.cuh"
#include "tc_common.cuh"

namespace goph {

using namespace tc;

// The preparation and the product of a call meet in scratch; `enqueue` is held from the one launch to the other, so
// that calls of several threads on one stream do not come between them.
struct QBufs {
  unsigned char* xb = nullptr;
  unsigned char* xaux = nullptr;
  float* xinv = nullptr;
  unsigned char* flags = nullptr;
  int* status = nullptr;
  size_t xb_bytes = 0;
  std::mutex enqueue;
};

namespace {

// Tuning build only (-DGOPH_TUNING): one CTA records clock64 at the hand-over points.
#ifdef GOPH_TUNING
__device__ long long g_qg_trace[8][64];
#define TP(...) __VA_ARGS__
#define MARK(ev, i) \
  if (blockIdx.x == gridDim.x / 2 && lane == 0 && (i) < 64) g_qg_trace[ev][i] = clock64()
#else
#define TP(...)
#define MARK(ev, i)
#endif

constexpr int kTileRows = 128;
constexpr int kChunkK = 256;
constexpr int kConvWarps = 16, kEpiWarps = 8, kEpiThreads = kEpiWarps * 32;  // in both pipes
constexpr int kWarpMMA = kConvWarps + kEpiWarps, kWarpB = kWarpMMA + 2, kWarpW = kWarpB + 1;  // two MMA warps
constexpr int kThreads = (kWarpW + 1) * 32;
// Registers: the block is launched with 72 a thread (896 threads: 64512); the epilogue, which keeps a
// row's sums of 64 columns, takes what the others give up: 256 * 128 + 512 * 48 + 128 * 56 = 64512.
// The compiler allots 72 to every role all the same and spills up to 160 bytes a thread in the epilogue's (frames of
// 8 to 40 bytes, the forms with two tiles most).
constexpr int kEpiRegs = 128, kConvRegs = 48, kMiscRegs = 56;
constexpr int kMaxSplits = 8;
constexpr int kMaxRows = 256;                       // activation rows of one launch

// What a format's slot of the weight ring looks like: [weights][row metadata].
template <int F, bool TILED>
struct QF {
  // packed nibbles in the row image (16-byte unit u of row r at r * 128 + ((u ^ (r & 7)) << 4)), else a
  // byte per weight as [16-byte unit][row] (tiled) or as two row images of 128 elements
  // (metadata beside them: kMeta bytes a row; Q6_K of the streaming layout: 16 of scales a row, then 4 with d a row)
  static constexpr bool kMLX = F == Q_MLX4 || F == Q_MLX4F;
  static constexpr bool kNibble = kMLX || F == Q_Q4K || (!TILED && (F == Q_Q5K || F == Q_Q6K));
  // Q5_K, Q6_K tiled: a nibble image in another order, and the bits above the nibbles beside it (mlx_mma.cu, Fmt)
  static constexpr bool kPacked = TILED && (F == Q_Q5K || F == Q_Q6K);
  static constexpr int kHigh = !kNibble && !kPacked ? 0 : F == Q_Q5K ? 4096 : F == Q_Q6K ? 8192 : 0;  // bits above the nibble, [16-byte unit][row]
  static constexpr int kHighOff = kTileRows * 128;
  static constexpr int kWBytes = (kNibble || kPacked ? kTileRows * 128 : kTileRows * 256) + kHigh;
  static constexpr int kMeta = F == Q_FP8 ? 0 : (F == Q_Q6K || F == Q_Q80) && !TILED ? 32 : 16;  // metadata bytes of a row
  static constexpr int kAux = F == Q_MLX4 ? 1 : F == Q_Q4K || F == Q_Q5K || F == Q_MLX4F ? 2 : 0;  // K16 steps of the affine term per chunk
  static constexpr bool kLong = F == Q_FP8 || F == Q_MLX4F;  // accumulator blocks of many chunks: nothing is scaled in between
  static constexpr bool kChunk = F == Q_Q4K || F == Q_Q5K;    // a block per pipe and chunk
  static constexpr int kBlk = F == Q_MLX4 ? 64 : F == Q_Q80 ? 32 : F == Q_Q6K ? 16 : 128;  // elements of a block, for the others
  static constexpr int kSlot = kWBytes + kTileRows * kMeta + (kPacked && F == Q_Q6K ? kTileRows * 2 : 0);  // (d behind the scales)
  static constexpr float kUnit = F == Q_MLX4 ? 16777216.f : F == Q_MLX4F ? 1.f / 1024.f : F == Q_Q4K || F == Q_Q5K ? 16384.f : 1.f;  // A holds the weights (the nibbles, the scale times the nibble) / kUnit
  // order of the elements inside a K16 step: 0 natural; 1 the nibble order (0 4 1 5 2 6 3 7 of each
  // packed word); 2 the same with the odd elements' activations scaled by 1/16
  static constexpr int kOrder = F == Q_MLX4 ? 2 : kNibble ? 1 : 0;
  // sums of x of the affine term: 1 four of 64 elements, 2 eight of 32, 3 four of 64 and eight times the same
  static constexpr int kSums = F == Q_MLX4 ? 1 : kChunk ? 2 : F == Q_MLX4F ? 3 : 0;
};

struct QArgs {
  const unsigned char* w;
  const void* aux;
  const unsigned char* xb;     // B tiles [row block][chunk * 2 + half][piece][K step 8][K half 2][n/8][8][16 B]
  const unsigned char* xaux;   // [row block][chunk][K16 step][K half 2][n/8][8][16 B]: sums of x in three bf16 pieces (scaled like x, / kUnit)
  const float* xinv;           // [batch] 2^-s of each activation row
  const unsigned char* flags;  // [row block][chunk][64] pieces in use, or nullptr: one piece
  const float* scale;
  const float* bias;
  float* out;
  int* status;
  size_t xb_stride;            // bytes of a row block in xb
  int out_dim, in_dim, batch;
  int ntiles, nchunks, nblocks;
  int nfull, ntail, splits;    // whole items (a multiple of the grid), then at most one per cluster, cut along K
  int dcol;                    // columns an accumulator block takes: 16, 32, 64 or 128
  int wslots, bslots, bslot, comb, pmax;  // depths of the rings, bytes of a B slot and of comb, pieces per half chunk in xb
};

// The row-major and streaming layouts' second argument: what load_rows asks for.  (Inside QArgs it also cost the tiled
// layouts' kernels registers: Q6_K 21504x1536 x256 129 us without, 136 with.)
struct QRowMaps {
  CUtensorMap map[3];
};
struct QNoMaps {};
template <bool TILED>
using QMapArgs = std::conditional_t<TILED, QNoMaps, QRowMaps>;

struct Walk {
  int k, tail, id, group, nb, split, c, c1, rot;
  bool live;
  __device__ __forceinline__ void open(const QArgs& a) {
    int j = k * (int)gridDim.x + (int)blockIdx.x;
    live = true;
    tail = -1;
    split = 0;
    if (j < a.nfull) {
      id = j;
      c = 0;
      c1 = a.nchunks;
    } else {
      // the CTAs of a cluster share the item (one each where nothing is cut), and it is their last
      j = (k - a.nfull / (int)gridDim.x) * (int)gridDim.x + (int)blockIdx.x;
      tail = j / a.splits;
      split = j - tail * a.splits;
      if (tail >= a.ntail) {
        live = false;
        return;
      }
      id = a.nfull + tail;
      c = split * a.nchunks / a.splits;
      c1 = (split + 1) * a.nchunks / a.splits;
    }
    group = id / a.nblocks;
    nb = id - group * a.nblocks;
    rot = (group * 5) % (c1 - c);
  }
  // The chunk to work on at step i of [c, c1): CTAs walk their K ranges in step, and starting every
  // group of tiles at a chunk of its own keeps them from all asking the L2 for the same activation
  // tile at the same moment.  (The sums are taken in this order; it is fixed per group.)
  __device__ __forceinline__ int chunk(int i) const { return i + rot < c1 ? i + rot : i + rot - (c1 - c); }
  __device__ __forceinline__ explicit Walk(const QArgs& a) : k(0) { open(a); }
  __device__ __forceinline__ void next_item(const QArgs& a) {
    ++k;
    open(a);
  }
};

template <int NB>
__device__ __forceinline__ int block_cols(const QArgs& a, int nb) {
  const int left = a.batch - nb * NB;
  return left >= NB ? NB : (left + 15) & ~15;
}

// ---- activation preparation -------------------------------------------------------------------

constexpr int kPrepThreads = 256;

__device__ __forceinline__ uint32_t f16_bits(float v) { return (uint32_t)__half_as_ushort(__float2half_rn(v)); }

// Grid (activation row, slice of its chunks): the row's largest magnitude, which every CTA of a row finds
// for itself (the row comes from the L2, four loads in flight per thread), then eight consecutive elements
// per thread and step, one 16-byte core-matrix row per piece; a warp covers one 256-element chunk per step.
template <int ORDER, int SUMS, bool XBF16>
__global__ void __launch_bounds__(kPrepThreads)
qg_prep_x_kernel(const void* __restrict__ xv, unsigned char* __restrict__ xb, unsigned char* __restrict__ xaux, float* __restrict__ xinv,
                 unsigned char* __restrict__ flags, int batch, int in_dim, int nchunks, int NB, size_t xb_stride, float unit_inv) {
  constexpr int P = XBF16 ? 1 : 3;
  __shared__ float red[kPrepThreads / 32];
  const int m = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
  const int nb = m / NB, j = m - nb * NB;
  pdl_launch_dependents();
  pdl_wait();  // x may be the output of the kernel in front; the tiles may still be read by it
  auto load8 = [&](int k, float (&v)[8]) {
    if (k >= in_dim) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.f;
    } else if (XBF16) {
      const uint4 q = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(xv) + (size_t)m * in_dim + k);
      const uint32_t ws[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[2 * e] = __uint_as_float(ws[e] << 16);
        v[2 * e + 1] = __uint_as_float(ws[e] & 0xFFFF0000u);
      }
    } else {
      const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(xv) + (size_t)m * in_dim + k);
      const float4 c = p[0], d = p[1];
      v[0] = c.x; v[1] = c.y; v[2] = c.z; v[3] = c.w;
      v[4] = d.x; v[5] = d.y; v[6] = d.z; v[7] = d.w;
    }
  };
  float mx = 0.f;
  for (int k = tid * 8; k < in_dim; k += 4 * kPrepThreads * 8) {
    float v[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) load8(k + i * kPrepThreads * 8, v[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int e = 0; e < 8; ++e) mx = fmaxf(mx, fabsf(v[i][e]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[tid >> 5] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int i = 1; i < kPrepThreads / 32; ++i) mx = fmaxf(mx, red[i]);
  // x * 2^s: the largest element lands in [2^14, 2^15)
  int E = (int)((__float_as_uint(mx) >> 23) & 0xFFu) - 127;
  // A row with an infinity: its outputs are infinite with the sign of the weight there (NaN for a zero weight or two
  // opposite ones) whatever the finite elements are, which only must not overflow an f16 themselves.
  if (mx == 0.f) E = 14;
  if (E > 127) E = 127;
  if (E < -112) E = -112;            // keeps 2^s a normal float
  const float s = __uint_as_float((uint32_t)(14 - E + 127) << 23);
  if (tid == 0 && blockIdx.y == 0) xinv[m] = __uint_as_float((uint32_t)(E - 14 + 127) << 23);
  int n = batch - nb * NB;
  n = n >= NB ? NB : (n + 15) & ~15;
  const int k_end = (int)((blockIdx.y + 1) * nchunks / gridDim.y) * kChunkK;
  for (int k = (int)(blockIdx.y * nchunks / gridDim.y) * kChunkK + tid * 8; k < k_end; k += kPrepThreads * 8) {
    float v[8];
    load8(k, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] *= s;
    const int c = k >> 8, half = (k >> 7) & 1, step = (k >> 4) & 7, kh = (k >> 3) & 1;
    if (SUMS != 0) {
      // sums of x per scale group, as three bf16 pieces (exact): slots [piece][sum] of the affine term's
      // K16 steps (four sums: 4 + 4 | 4 and zeros; eight: 8 | 8, then 8 | zeros)
      constexpr int kG = SUMS == 1 ? 4 : 8, kPer = SUMS == 2 ? 4 : 8, kSteps = SUMS == 1 ? 1 : 2;
      float t = ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
      t += __shfl_xor_sync(0xffffffffu, t, 1);
      t += __shfl_xor_sync(0xffffffffu, t, 2);
      if (SUMS != 2) t += __shfl_xor_sync(0xffffffffu, t, 4);
      t *= unit_inv;
      uint32_t piece[3];
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        piece[p] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(t));
        t -= __uint_as_float(piece[p] << 16);
      }
      // lane l gathers slot l (of 16 or 32): sum l % kG, piece l / kG
      const int src = (SUMS == 3 ? lane % 4 : lane % kG) * kPer;
      const uint32_t g0 = __shfl_sync(0xffffffffu, piece[0], src), g1 = __shfl_sync(0xffffffffu, piece[1], src),
                     g2 = __shfl_sync(0xffffffffu, piece[2], src);
      const int pc = lane / kG;
      uint32_t mine = pc == 0 ? g0 : pc == 1 ? g1 : pc == 2 ? g2 : 0u;
      if (SUMS == 3 && (lane & 4)) mine = __float_as_uint(__uint_as_float(mine << 16) * 8.f) >> 16;  // exact
      if (lane < 16 * kSteps)
        *reinterpret_cast<unsigned short*>(xaux + ((size_t)nb * nchunks + c) * (kSteps * 32) * NB + (lane >> 4) * (n * 32) + ((lane >> 3) & 1) * (n * 16) +
                                           (j >> 3) * 128 + (j & 7) * 16 + (lane & 7) * 2) = (unsigned short)mine;
    }
    if (ORDER == 2) {
#pragma unroll
      for (int e = 1; e < 8; e += 2) v[e] *= 0.0625f;
    }
    unsigned char* dst = xb + (size_t)nb * xb_stride + (size_t)(c * 2 + half) * P * n * 256 + step * (n * 32) + kh * (n * 16) + (j >> 3) * 128 + (j & 7) * 16;
    int used = 1;
#pragma unroll
    for (int p = 0; p < P; ++p) {
      uint32_t h[8], any = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        h[e] = f16_bits(v[e]);
        any |= h[e] & 0x7FFFu;
        v[e] -= __half2float(__ushort_as_half((unsigned short)h[e]));  // exact
        if ((h[e] & 0x7FFFu) >= 0x7C00u) v[e] = 0.f;                   // (and not inf - inf)
      }
      uint32_t q[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) q[ORDER == 0 ? e : 2 * (e & 3) + (e >> 2)] = h[e];
      *reinterpret_cast<uint4*>(dst + (size_t)p * n * 256) =
          make_uint4(q[0] | (q[1] << 16), q[2] | (q[3] << 16), q[4] | (q[5] << 16), q[6] | (q[7] << 16));
      if (P > 1 && p > 0 && __any_sync(0xffffffffu, any != 0)) used = p + 1;
    }
    if (P > 1 && lane == 0) flags[((size_t)nb * nchunks + c) * 64 + j] = (unsigned char)used;
  }
}

// ---- the product kernel: pieces ------------------------------------------------------------------

__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t fma2h(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

template <int N>
__device__ __forceinline__ void reg_dec() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void reg_inc() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// Box of a two-dimensional tensor map at byte x of row y.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y),
               "r"(bar)
               : "memory");
}

// The row-major and streaming layouts: one chunk of one tile into a slot, by a warp.  Weights come as boxes of 128 rows x
// 128 bytes, whose 128-byte swizzle is the row image's (16-byte unit u of row r at r * 128 + ((u ^ (r & 7)) << 4)), what
// stands between or beside them as boxes of 128 rows x 16 bytes; every x is a multiple of 16.  Only the f16 scales of
// Q6_K and Q8_0 come by cp.async (an MLX table whose rows are no whole 16-byte units is copied once, at upload; by cp.async 5018x15424 x8 33.0 us, so 24.1, 3000x4160 x30 15.5 and 13.3).  (One warp's cp.async of
// everything, 44 to 72 a chunk with their addresses, set the pace: B200, us a call, Q5_K 489x9728 x93 39.6 -> 22.7, Q8_0
// 11376x1504 x42 28.5 -> 23.3, Q6_K 1024x1792 x29 21.4 -> 11.2, FP8 2816x3136 x5 12.3 -> 9.4, MLX4 5722x1280 x99 16.1 -> 12.8.)
template <int F>
__device__ __forceinline__ bool rows_cp(const QRowMaps& t) {  // whether a chunk has a part for cp.async
  return F == Q_Q6K || F == Q_Q80;
}
template <int F>
__device__ __forceinline__ void load_rows(const QArgs& a, const QRowMaps& t, uint32_t slot, uint32_t bar, int tile, int c, int lane) {
  typedef QF<F, false> T;
  const int row0 = tile * kTileRows;
  const uint32_t meta = slot + T::kWBytes;
  if (lane == 0) {
    constexpr uint32_t kBytes = T::kWBytes + (F == Q_Q80 || F == Q_FP8 ? 0 : 2048);
    mbar_expect_tx(bar, kBytes);
    if (T::kMLX) {
      tma_load_2d(slot, &t.map[0], c * 128, row0, bar);
      tma_load_2d(meta, &t.map[1], c * 16, row0, bar);
    } else if (F == Q_Q4K || F == Q_Q5K) {  // super-blocks {16-byte header, nibbles, Q5_K: fifth bits}
      const int x = c * (F == Q_Q4K ? 144 : 176);
      tma_load_2d(slot, &t.map[0], x + 16, row0, bar);
      tma_load_2d(meta, &t.map[1], x, row0, bar);
      if (F == Q_Q5K) {
        tma_load_2d(slot + T::kHighOff, &t.map[1], x + 144, row0, bar);
        tma_load_2d(slot + T::kHighOff + 2048, &t.map[1], x + 160, row0, bar);
      }
    } else if (F == Q_Q6K) {  // planes: low nibbles, highs, scales
      tma_load_2d(slot, &t.map[0], c * 128, row0, bar);
#pragma unroll
      for (int u = 0; u < 4; ++u) tma_load_2d(slot + T::kHighOff + u * 2048, &t.map[1], c * 64 + 16 * u, row0, bar);
      tma_load_2d(meta, &t.map[2], c * 16, row0, bar);
    } else {  // a byte per weight
      tma_load_2d(slot, &t.map[0], c * 256, row0, bar);
      tma_load_2d(slot + 16384, &t.map[0], c * 256 + 128, row0, bar);
    }
  }
  __syncwarp();
  if (F == Q_Q6K) {  // the f16 d, in its aligned pair (the last one of an odd count stands alone)
    const unsigned char* dd = static_cast<const unsigned char*>(a.aux) + (size_t)a.out_dim * a.in_dim / 4 + (size_t)a.out_dim * a.in_dim / 16;
    const size_t total = (size_t)a.out_dim * a.nchunks;
    for (int r = lane; r < 128; r += 32) {
      const bool ok = row0 + r < a.out_dim;
      const size_t word = ((size_t)(ok ? row0 + r : 0) * a.nchunks + c) >> 1;
      cp_async4(meta + 2048 + r * 4, dd + word * 4, !ok ? 0 : 2 * word + 1 < total ? 4 : 2);
    }
  } else if (F == Q_Q80) {  // the row's f16 scales from the aligned pair that holds the first one
    const int nb = a.in_dim / 32;
    const size_t total = (size_t)a.out_dim * nb;
    const unsigned char* d = static_cast<const unsigned char*>(a.aux);
    for (int r = lane; r < 128; r += 32) {
      const size_t word = ((size_t)(row0 + r) * nb + c * 8) >> 1;
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const bool ok = row0 + r < a.out_dim && 2 * (word + k) < total;
        cp_async4(meta + r * 32 + k * 4, ok ? d + (word + k) * 4 : d, !ok ? 0 : 2 * (word + k) + 1 < total ? 4 : 2);
      }
    }
  }
}

// Field of sub-block s (0..7, a constant after unrolling) of a K-quant header: scale | minimum << 6.
__device__ __forceinline__ uint32_t kq_field(const uint4& h, int s) {
  const int bit = 12 * s, wi = bit >> 5, sh = bit & 31;
  const uint32_t lo = wi == 0 ? h.y : wi == 1 ? h.z : h.w;
  const uint32_t hi = wi == 0 ? h.z : wi == 1 ? h.w : 0u;
  return __funnelshift_r(lo, hi, sh) & 0xFFFu;
}
// The 6-bit scale as a pair of f16: times 2^10 (exact, at most 64512).
__device__ __forceinline__ uint32_t kq_scale2(uint32_t field) {
  const uint32_t v = field & 63u;
  return mul2(sub2((v | (v << 16)) | 0x64006400u, 0x64006400u), 0x64006400u);
}

// 64 elements (quarter kq of half hh of the chunk) of row r: f16 values into the A buffer's columns at `abuf`.
template <int F, bool TILED>
__device__ __forceinline__ void convert_unit(const unsigned char* st, int r, int hh, int kq, uint32_t abuf) {
  typedef QF<F, TILED> T;
  uint4 head = make_uint4(0, 0, 0, 0);
  if (F == Q_Q4K || F == Q_Q5K) head = *reinterpret_cast<const uint4*>(st + T::kWBytes + r * 16);
  const int u0 = 4 * hh + 2 * kq;  // the first of two 32-element sub-blocks
  uint32_t fs = 0;                 // MLX4F: the group's scale times 2^10, as a pair of f16 (exact)
  if (F == Q_MLX4F) {
    const uint32_t m = *reinterpret_cast<const uint32_t*>(st + T::kWBytes + r * 16 + (2 * hh + kq) * 4);
    fs = f16_bits(__uint_as_float(m << 16) * 1024.f);
    fs |= fs << 16;
  }
  if (T::kNibble) {
    uint4 qv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) qv[u] = *reinterpret_cast<const uint4*>(st + r * 128 + (((u0 + u) ^ (r & 7)) << 4));
    uint2 hb = make_uint2(0, 0);       // Q5_K: fifth bits, a word per 32 elements
    uint4 hv = make_uint4(0, 0, 0, 0);  // Q6_K: two bits per element, two words per 32
    if (F == Q_Q5K) hb = *reinterpret_cast<const uint2*>(st + T::kHighOff + hh * 2048 + r * 16 + kq * 8);
    if (F == Q_Q6K) hv = *reinterpret_cast<const uint4*>(st + T::kHighOff + (2 * hh + kq) * 2048 + r * 16);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t ws[4] = {qv[u].x, qv[u].y, qv[u].z, qv[u].w};
      uint32_t m0 = 0, m1 = 0;  // Q4_K, Q5_K: the sub-block's scale for nibbles read as n and as 16 n
      if (F == Q_Q4K || F == Q_Q5K) {
        m0 = kq_scale2(kq_field(head, u0 + u));
        m1 = mul2(m0, 0x2C002C00u);  // / 16
      }
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {
        uint32_t regs[8];
#pragma unroll
        for (int wi = 0; wi < 2; ++wi) {
          const uint32_t w = ws[2 * s2 + wi], w8 = w >> 8;
          uint32_t e[4] = {w & 0x000F000Fu, w & 0x00F000F0u, w8 & 0x000F000Fu, w8 & 0x00F000F0u};
          if (F == Q_MLX4F) {
            // (n - 8) times the scale: 4 + 8 bits less one, exact
            e[0] = mul2(sub2(e[0] | 0x64006400u, 0x64086408u), fs);               // 1024 + n
            e[1] = mul2(fma2h(e[1] | 0x64006400u, 0x2C002C00u, 0xD480D480u), fs);  // (1024 + 16 n) / 16 - 72
            e[2] = mul2(sub2(e[2] | 0x64006400u, 0x64086408u), fs);
            e[3] = mul2(fma2h(e[3] | 0x64006400u, 0x2C002C00u, 0xD480D480u), fs);
          } else if (F == Q_Q4K) {
            e[0] = mul2(e[0], m0);
            e[1] = mul2(e[1], m1);
            e[2] = mul2(e[2], m0);
            e[3] = mul2(e[3], m1);
          } else if (F == Q_Q5K) {
            // fifth bits of the word's eight elements, those of 0..3 in the low half and of 4..7 in the high half
            const uint32_t b8 = ((u == 0 ? hb.x : hb.y) >> (8 * (2 * s2 + wi))) & 0xFFu, t = (b8 & 0xFu) | ((b8 >> 4) << 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t n = (k & 1) ? e[k] >> 4 : e[k];
              e[k] = mul2(n | (((t >> k) & 0x00010001u) << 4), m0);
            }
          } else if (F == Q_Q6K) {
            // two bits of the word's eight elements: 0..3 in the low half, 4..7 in the high half
            const uint32_t hw = u == 0 ? (s2 == 0 ? hv.x : hv.y) : (s2 == 0 ? hv.z : hv.w);
            const uint32_t h16 = (hw >> (16 * wi)) & 0xFFFFu, t = (h16 & 0xFFu) | ((h16 >> 8) << 16);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const uint32_t n = (k & 1) ? e[k] >> 4 : e[k];
              e[k] = sub2(n | (((t >> (2 * k)) & 0x00030003u) << 4) | 0x64006400u, 0x64206420u);  // (1024 + q) - 1056
            }
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) regs[4 * wi + k] = e[k];
        }
        tmem_st8(abuf + (2 * u + s2) * 8, regs);
      }
    }
  } else if (T::kPacked) {
    uint4 qv[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) qv[u] = *reinterpret_cast<const uint4*>(st + r * 128 + (((u0 + u) ^ (r & 7)) << 4));
    const uint4 hv = *reinterpret_cast<const uint4*>(st + T::kHighOff + (F == Q_Q6K ? 2 * hh + kq : hh) * 2048 + r * 16);
    const uint32_t hs[4] = {hv.x, hv.y, hv.z, hv.w};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t ws[4] = {qv[u].x, qv[u].y, qv[u].z, qv[u].w};
      uint32_t m0 = 0;
      if (F == Q_Q5K) m0 = kq_scale2(kq_field(head, u0 + u));
#pragma unroll
      for (int s2 = 0; s2 < 2; ++s2) {  // the unit's first 16 elements are the low nibbles, the others the high ones
        uint32_t regs[8];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const int f = (F == Q_Q6K ? 2 * u : 4 * kq + 2 * u) + s2;  // the field in the bits' bytes
          uint32_t w = (s2 ? ws[t] >> 4 : ws[t]) & 0x0F0F0F0Fu;
          if (F == Q_Q6K) {
            w |= (f < 2 ? hs[t] << (4 - 2 * f) : hs[t] >> (2 * f - 4)) & 0x30303030u;
            regs[2 * t] = sub2(__byte_perm(w, 0x64646464u, 0x4140), 0x64206420u);  // (1024 + q) - 1056
            regs[2 * t + 1] = sub2(__byte_perm(w, 0x64646464u, 0x4342), 0x64206420u);
          } else {
            w |= (f < 4 ? hs[t] << (4 - f) : hs[t] >> (f - 4)) & 0x10101010u;
            regs[2 * t] = mul2(__byte_perm(w, 0u, 0x4140), m0);
            regs[2 * t + 1] = mul2(__byte_perm(w, 0u, 0x4342), m0);
          }
        }
        tmem_st8(abuf + (2 * u + s2) * 8, regs);
      }
    }
  } else {
    uint4 qv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      qv[u] = *reinterpret_cast<const uint4*>(TILED ? st + (8 * hh + 4 * kq + u) * 2048 + r * 16 : st + hh * 16384 + r * 128 + (((4 * kq + u) ^ (r & 7)) << 4));
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t ws[4] = {qv[u].x, qv[u].y, qv[u].z, qv[u].w};
      uint32_t regs[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t w = ws[k];
        if (F == Q_FP8) {
          asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(regs[2 * k]) : "h"((unsigned short)(w & 0xFFFFu)));
          asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(regs[2 * k + 1]) : "h"((unsigned short)(w >> 16)));
        } else {
          if (TILED) w ^= 0x80808080u;  // signed bytes; the streaming layout keeps q + 128
          regs[2 * k] = sub2(__byte_perm(w, 0x64646464u, 0x4140), 0x64806480u);  // (1024 + 128 + q) - 1152
          regs[2 * k + 1] = sub2(__byte_perm(w, 0x64646464u, 0x4342), 0x64806480u);
        }
      }
      tmem_st8(abuf + u * 8, regs);
    }
  }
}

// The affine term's A operand of row r: the chunk's biases (MLX4: four, twice; MLX4F: four biases and the
// four scales that meet the 8 taken from every nibble) or minima (K-quants: eight) as eight bf16, in both
// K halves of a K16 step.
template <int F, bool TILED>
__device__ __forceinline__ void convert_aux(const unsigned char* st, int r, unsigned char* dst) {
  const uint4 h = *reinterpret_cast<const uint4*>(st + QF<F, TILED>::kWBytes + r * 16);
  uint4 v;
  if (F == Q_MLX4) {
    v.x = v.z = __byte_perm(h.x, h.y, 0x7632);
    v.y = v.w = __byte_perm(h.z, h.w, 0x7632);
  } else if (F == Q_MLX4F) {
    v.x = __byte_perm(h.x, h.y, 0x7632);
    v.y = __byte_perm(h.z, h.w, 0x7632);
    v.z = __byte_perm(h.x, h.y, 0x5410);
    v.w = __byte_perm(h.z, h.w, 0x5410);
  } else {
    uint32_t b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // small integers are exact in bf16
      const uint32_t lo = __float_as_uint((float)(kq_field(h, 2 * k) >> 6)), hi = __float_as_uint((float)(kq_field(h, 2 * k + 1) >> 6));
      b[k] = (lo >> 16) | (hi & 0xFFFF0000u);
    }
    v = make_uint4(b[0], b[1], b[2], b[3]);
  }
  unsigned char* d = dst + (r >> 3) * 128 + (r & 7) * 16;
  *reinterpret_cast<uint4*>(d) = v;
  *reinterpret_cast<uint4*>(d + 2048) = v;
}
// D[tmem] (+)= A[tmem] * B[smem descriptor: low and high word], 16-bit floats, f32 accumulate.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "mov.b64 b, {%2, %3};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
      : "memory");
}
// D[tmem] (+)= A[smem descriptor] * B[smem descriptor], 16-bit floats, f32 accumulate.
__device__ __forceinline__ void umma_f16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}

// ---- the product kernel ----------------------------------------------------------------------------
// TT: row tiles of an item; NB: activation rows of an item (columns of an accumulator block).
// The work runs in two pipes, each with its converters, MMA warp, accumulators and epilogue warps: a
// pipe takes one of the two tiles (TT = 2), or one half of every chunk (TT = 1; their sums meet in
// shared memory when the item ends).  One issuing warp alone could not keep up: a wait that succeeds at
// once still costs it over a hundred cycles, and an MMA forty.
template <int F, bool TILED, int TT, int NB>
__global__ void __launch_bounds__(kThreads, 1)
qg_kernel(const __grid_constant__ QArgs a, const __grid_constant__ QMapArgs<TILED> maps) {
  typedef QF<F, TILED> T;
  static_assert(NB == 64 || (NB == 128 && F == Q_FP8 && TT == 2), "wide blocks only where a block is read once per item");
  constexpr bool kLong = T::kLong, kChunk = T::kChunk;
  constexpr bool kItemBlock = kLong && NB == 128; // one per item, read straight to the result
  // The tensor core's f32 sums drift towards zero with their length (0.6e-6 of the largest output at 8192
  // elements): a block is closed and added in registers every 4096, an item of one block is kept to 8192
  constexpr int kSeg = kItemBlock ? 1 << 20 : 16;
  constexpr int kAB = kLong && NB == 64 ? 3 : 2;  // A units (128 elements, 64 TMEM columns) of a pipe
  constexpr int kDC = 256 - kAB * 64;             // accumulator columns of a pipe: DT blocks of a.dcol
  constexpr int kPer = kLong || kChunk ? 1 : 128 / T::kBlk; // blocks (or the part of one) in a unit
  constexpr int KS = 8 / kPer;                    // K16 steps of it
  constexpr int UPC = TT == 2 ? 2 : 1;            // units a pipe takes of a chunk
  constexpr int UB = kLong ? kSeg * UPC : kChunk ? UPC : 1;  // units of a block
  constexpr int kAuxBytes = T::kAux ? 2 * kAB * 4096 : 0;  // the affine term's A operand, one beside each A unit
  constexpr uint32_t kCols = 512;

  extern __shared__ unsigned char smem_dyn[];
  unsigned char* wring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  const int SW = a.wslots, SB = a.bslots, DT = kDC / a.dcol;
  unsigned char* bring = wring + (size_t)SW * T::kSlot;
  unsigned char* aux = bring + (size_t)SB * a.bslot;
  float* comb = reinterpret_cast<float*>(aux + kAuxBytes);  // TT = 1: [column][128] sums of pipe 1
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(comb) + (TT == 1 ? a.comb : 0));
  const uint32_t wfull = smem_u32(bars), wempty = wfull + 8 * SW, bfull = wempty + 8 * SW, bempty = bfull + 8 * SB;
  const uint32_t aready = bempty + 8 * SB, afree = aready + 64, dfull = afree + 64, dfree = dfull + 128;  // [pipe][4], [pipe][8]
  volatile int* pieces = reinterpret_cast<volatile int*>(bars + 2 * SW + 2 * SB + 48);  // [SB] pieces in the slot
  uint32_t* tmem_holder = const_cast<uint32_t*>(reinterpret_cast<volatile uint32_t*>(pieces + SB));
  float* xinv = reinterpret_cast<float*>(tmem_holder + 1);  // [kMaxRows]
  volatile int* shared_item = reinterpret_cast<volatile int*>(xinv + kMaxRows);  // the cluster's item: group (or -1), block, split

  // (the shuffle tells the compiler that a warp's number is the same in all of its lanes: what follows from it is
  // kept in uniform registers, from where the MMAs take their operands.  Q8_0 4096x4096 x19 16.5 us without, 15.1
  // with, Q4_K 14336x4096 x64 30.8 and 29.4)
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  Walk wk(a);
  auto load_weights = [&](int s, int t, int c) {  // the W loader: chunk c of the item's tile t into slot s
    int tile = wk.group * TT + t;
    if (tile >= a.ntiles) tile = a.ntiles - 1;  // the last group of an odd tile count repeats its tile (nothing of the copy is stored)
    const uint32_t slot = smem_u32(wring) + s * T::kSlot;
    if constexpr (!TILED) {
      load_rows<F>(a, maps, slot, wfull + 8 * s, tile, c, lane);
      if (rows_cp<F>(maps)) cp_async_arrive(wfull + 8 * s);
    } else if (lane == 0) {
      mbar_expect_tx(wfull + 8 * s, T::kSlot);
      bulk_load_1d(slot, a.w + ((size_t)tile * a.nchunks + c) * T::kSlot, T::kSlot, wfull + 8 * s);
    }
  };
  // The set-up, spread over four warps (by one thread it took 1.7 us with what follows it): the first two
  // weight stages, which do not depend on the kernel in front, are asked for before anything else.
  const int early = !wk.live ? 0 : TT == 2 || wk.c + 1 < wk.c1 ? 2 : 1;
  if (warp == kWarpW) {
    if (lane < SW) {
      int arrivals = 1;
      if constexpr (!TILED) arrivals += rows_cp<F>(maps) ? 32 : 0;
      mbar_init(wfull + 8 * lane, arrivals);
      mbar_init(wempty + 8 * lane, TT == 2 ? 8 + (kLong ? 0 : 4) : 2 * (4 + (kLong ? 0 : 4)));
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    for (int i = 0; i < early; ++i) load_weights(i, TT == 2 ? i : 0, wk.chunk(TT == 2 ? wk.c : wk.c + i));
  } else if (warp == kWarpB) {
    if (lane < SB) {
      mbar_init(bfull + 8 * lane, 1);
      mbar_init(bempty + 8 * lane, TT);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  } else if (warp == kWarpMMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)), "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  } else if (warp == kWarpMMA + 1) {
    if (lane < 8) {
      mbar_init(aready + 8 * lane, 4);
      mbar_init(afree + 8 * lane, 1);
    } else if (lane < 24) {
      mbar_init(dfull + 8 * (lane - 8), 1);
      mbar_init(dfree + 8 * (lane - 8), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;  // A: columns [pipe][kAB][64], then D: [pipe][DT][a.dcol]
  bool ok = true;
  // is the affine term of the item's i-th chunk this pipe's, and with which unit of the chunk
  auto aux_here = [&](int w, int i, int u) { return T::kAux != 0 && (TT == 2 ? u == 1 : (i & 1) == w); };

  if (warp == kWarpW) {
    // ------------------------------------------------------------------ weights
    reg_dec<kMiscRegs>();
    if (!TILED || lane == 0) {
      RingCursor cur;
      int i = 0;
      for (; wk.live && ok; wk.next_item(a)) {
        for (int ci = wk.c; ci < wk.c1 && ok; ++ci) {
          const int c = wk.chunk(ci);
#pragma unroll 1
          for (int t = 0; t < TT; ++t, ++i, cur.next(SW)) {
            // The first two stages have been asked for, the rest of the ring follows when the first is in (a
            // grid that asked for all its rings at once would see every first stage land last).
            if (i < early) continue;
            if (i == early) ok = mbar_wait(wfull, 0, a.status, 801);
            if (ok && i >= SW) ok = mbar_wait(wempty + 8 * cur.s, cur.ph ^ 1u, a.status, 802);
            // (load_rows is for whole warps: lanes that disagree, one at its limit, one just released, must not part)
            if (!TILED) ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (lane == 0) { MARK(0, i); }
            load_weights(cur.s, t, c);
          }
        }
      }
    }
    if (!TILED) asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  } else if (warp == kWarpB) {
    // ------------------------------------------------------------------ prepared activations
    reg_dec<kMiscRegs>();
    pdl_wait();
    MARK(7, 0);
    RingCursor bc;
    bool wrapped = false;
    auto used_of = [&](const Walk& w, int c) -> uint32_t {  // most pieces any of the block's rows has in this chunk
      if (!a.flags) return 1u;
      const unsigned char* f = a.flags + ((size_t)w.nb * a.nchunks + c) * 64;
      const int col = w.nb * NB + 2 * lane;
      uint32_t v = 1;
      if (col < a.batch) v = max(v, (uint32_t)__ldcg(f + 2 * lane));
      if (col + 1 < a.batch) v = max(v, (uint32_t)__ldcg(f + 2 * lane + 1));
      return v;
    };
    auto load_half = [&](int s, int ci, int h, int P) {  // half chunk h of the item's step ci, P pieces; returns the bytes
      const int n = block_cols<NB>(a, wk.nb), c = wk.chunk(ci);
      const uint32_t bytes = n * 256, axb = T::kAux * n * 32, dst = smem_u32(bring) + s * a.bslot;  // bytes: of a piece
      bulk_load_1d(dst, a.xb + (size_t)wk.nb * a.xb_stride + (size_t)(2 * c + h) * a.pmax * bytes, P * bytes, bfull + 8 * s);
      const bool ax = TT == 2 ? aux_here(0, 0, h) : aux_here(h, ci - wk.c, 0);
      if (ax) bulk_load_1d(dst + a.pmax * bytes, a.xaux + ((size_t)wk.nb * a.nchunks + c) * (T::kAux * 32 * NB), axb, bfull + 8 * s);
      return P * bytes + (ax ? axb : 0);
    };
    // the first two half chunks come whole, so that they need not wait for the flags
    uint32_t first0 = 0, first1 = 0;
    if (wk.live && lane == 0) {
      first0 = load_half(0, wk.c, 0, a.pmax);
      first1 = load_half(1, wk.c, 1, a.pmax);
    }
    bool first = true;
    for (; wk.live && ok; wk.next_item(a)) {
      uint32_t nxt = used_of(wk, wk.chunk(wk.c));
      for (int ci = wk.c; ci < wk.c1 && ok; ++ci) {
        const uint32_t cur = nxt;
        if (ci + 1 < wk.c1) nxt = used_of(wk, wk.chunk(ci + 1));
        const int P = (int)__reduce_max_sync(0xffffffffu, cur);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int s = bc.s;
          if (wrapped) ok = __all_sync(0xffffffffu, mbar_wait(bempty + 8 * s, bc.ph ^ 1u, a.status, 803));
          if (!ok) break;
          if (lane == 0) {
            pieces[s] = P;
            const uint32_t bytes = first ? (h ? first1 : first0) : load_half(s, ci, h, P);
            mbar_expect_tx(bfull + 8 * s, bytes);
          }
          __syncwarp();
          bc.next(SB);
          wrapped = wrapped || bc.s == 0;
        }
        first = false;
      }
    }
  } else if (warp >= kWarpMMA) {
    // ------------------------------------------------------------------ MMA, a warp per pipe
    reg_dec<kMiscRegs>();
    const int w = warp - kWarpMMA;
    RingCursor bc, ac, dc;  // B slots, A buffers (kAB), accumulator blocks (DT)
    int used = 0;           // accumulator blocks opened so far, up to DT
    if (TT == 1 && w == 1) bc.next(SB);
    // (the masks: in a cluster launch a shared-memory address carries the CTA's rank above the 18 bits that descriptors hold)
    const uint32_t bring_u = (smem_u32(bring) >> 4) & 0x3FFF, ar = aready + 32 * w, af = afree + 32 * w, df = dfull + 64 * w, de = dfree + 64 * w;
    const uint32_t colA = tmem + w * (kAB * 64), colD = tmem + 2 * kAB * 64 + w * kDC;
    TP(int mk = 0;)
    // the next accumulator block is free (the epilogue has read what it held)
    auto open_block = [&] {
      if (used < DT) {
        ++used;
        return true;
      }
      const bool r = __all_sync(0xffffffffu, mbar_wait(de + 8 * dc.s, dc.ph ^ 1u, a.status, 807));
      tc_fence_after();
      return r;
    };
    for (; wk.live && ok; wk.next_item(a)) {
      const int n = block_cols<NB>(a, wk.nb);
      // instruction descriptor: D f32, A f16, B f16, both K-major, N = n, M = 128; the affine term's: A, B bf16
      const uint32_t idesc = (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24), idesc_aux = idesc | (1u << 7) | (1u << 10);
      // B descriptors: halves n * 16 B apart, row groups 128 B; address and the first stride in the low word
      const uint32_t dlo = bring_u | ((uint32_t)n << 16), bhi = (128u >> 4) | (1u << 14), n2 = n * 2;
      const int units = (wk.c1 - wk.c) * UPC;
      for (int i = 0; i < units; ++i) {
        ok = mbar_wait(bfull + 8 * bc.s, bc.ph, a.status, 804) && mbar_wait(ar + 8 * ac.s, ac.ph, a.status, 806);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        if (w == 0) { MARK(3, mk); }
        const int P = pieces[bc.s];
        const uint32_t blo = dlo + ((bc.s * a.bslot) >> 4), acol = colA + ac.s * 64;
        const bool opens = UB == 1 || i % UB == 0, closes = UB == 1 || i + 1 == units || (i + 1) % UB == 0;
        const bool ax = aux_here(w, i / UPC, i % UPC);
        const uint64_t adesc = ((uint64_t)(2048u >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46) | (uint64_t)((smem_u32(aux + (w * kAB + ac.s) * 4096) >> 4) & 0x3FFF);
#pragma unroll
        for (int b = 0; b < kPer; ++b) {
          if (opens) {
            ok = open_block();
            if (!ok) break;
          }
          if (elect_one()) {
            const uint32_t dcol = colD + dc.s * a.dcol;
#pragma unroll
            for (int p = 0; p < 3; ++p) {
              if (p < P) {
#pragma unroll
                for (int k = 0; k < KS; ++k)
                  umma_f16_ts(dcol, acol + (b * KS + k) * 8, blo + (p * 8 + b * KS + k) * n2, bhi, idesc, !(opens && p == 0 && k == 0));
              }
            }
            if (kLong && T::kAux != 0 && ax) {  // the affine term joins the open block
#pragma unroll
              for (int k = 0; k < T::kAux; ++k) umma_f16_ss(dcol, adesc, ((uint64_t)bhi << 32) | (blo + a.pmax * (n * 16) + k * n2), idesc_aux, 1);
            }
            if (closes) umma_commit(df + 8 * dc.s);
          }
          __syncwarp();
          if (closes) dc.next(DT);
        }
        if (!ok) break;
        if (!kLong && T::kAux != 0 && ax) {
          ok = open_block();
          if (!ok) break;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < T::kAux; ++k)
              umma_f16_ss(colD + dc.s * a.dcol, adesc, ((uint64_t)bhi << 32) | (blo + a.pmax * (n * 16) + k * n2), idesc_aux, k != 0);
            umma_commit(df + 8 * dc.s);
          }
          __syncwarp();
          dc.next(DT);
        }
        if (elect_one()) {
          umma_commit(af + 8 * ac.s);
          umma_commit(bempty + 8 * bc.s);
        }
        __syncwarp();
        if (w == 0) { MARK(4, mk); }
        TP(++mk;)
        ac.next(kAB);
        bc.next(SB);
        if (TT == 1) bc.next(SB);
      }
    }
  } else if (warp < kConvWarps) {
    // ------------------------------------------------------------------ converters, two groups of four warps per pipe
    // The groups take turns at the pipe's units, thread = row: while one waits, stores and hands over (some
    // 500 cycles of a unit), the other converts.
    reg_dec<kConvRegs>();
    const int w = warp >> 3, grp = (warp >> 2) & 1, q4 = warp & 3, r = q4 * 32 + lane;
    RingCursor wc, ac;
    bool used = false;  // this A buffer has been filled before
    int cc = 0;         // chunks so far
    if (TT == 2 && w == 1) wc.next(SW);
    if (grp == 1) ac.next(kAB);
    const uint32_t abase = tmem + ((uint32_t)(q4 * 32) << 16) + w * (kAB * 64), ar = aready + 32 * w, af = afree + 32 * w;
    TP(int mk = 0;)
    for (; wk.live && ok; wk.next_item(a)) {
      for (int ci = wk.c; ci < wk.c1 && ok; ++ci, ++cc) {
        if (TT == 2 || (cc & 1) == grp) {
          ok = __all_sync(0xffffffffu, mbar_wait(wfull + 8 * wc.s, wc.ph, a.status, 808));
          if (ok && used) ok = __all_sync(0xffffffffu, mbar_wait(af + 8 * ac.s, ac.ph ^ 1u, a.status, 809));
          if (!ok) break;
          tc_fence_after();
          if (warp == 0) { MARK(1, mk); }
          const unsigned char* st = wring + wc.s * T::kSlot;
          if (aux_here(w, ci - wk.c, grp)) {
            convert_aux<F, TILED>(st, r, aux + (w * kAB + ac.s) * 4096);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMA reads it through the async proxy
          }
          convert_unit<F, TILED>(st, r, TT == 2 ? grp : w, 0, abase + ac.s * 64);
          convert_unit<F, TILED>(st, r, TT == 2 ? grp : w, 1, abase + ac.s * 64 + 32);
          __syncwarp();
          if (lane == 0) mbar_arrive(wempty + 8 * wc.s);
          tmem_wait_st();
          tc_fence_before();
          warp_arrive(ar + 8 * ac.s, lane);
          if (warp == 0) { MARK(2, mk); }
          TP(++mk;)
          ac.next(kAB);
          used = used || ac.ph != 0;
          ac.next(kAB);
          used = used || ac.ph != 0;
        }
        wc.next(SW);
        if (TT == 2) wc.next(SW);
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue, four warps per pipe: a row's NB columns per thread
    reg_inc<kEpiRegs>();
    const int e = warp - kConvWarps, q4 = warp & 3, w = e >> 2;
    const int r = q4 * 32 + lane, t = TT == 2 ? w : 0;
    const uint32_t dbase = tmem + 2 * kAB * 64 + ((uint32_t)(q4 * 32) << 16) + w * kDC, df = dfull + 64 * w, de = dfree + 64 * w;
    RingCursor wc, dc;
    if (TT == 2 && w == 1) wc.next(SW);
    TP(int mk = 0;)
    float2 acc[kItemBlock ? 1 : NB / 2];
    // TT = 1: the pipes' sums meet through shared memory; afterwards a pipe holds every other group of four columns
    auto combine = [&](int n) {
      if constexpr (TT == 1 && !kItemBlock) {
        float4* cb = reinterpret_cast<float4*>(comb) + r;
#pragma unroll
        for (int g = 0; g < NB / 4; ++g) {
          if (4 * g >= n) break;  // (out of the unrolled loop: a step over each group costs an instruction fetch)
          if ((g & 1) != w) cb[g * kTileRows] = make_float4(acc[2 * g].x, acc[2 * g].y, acc[2 * g + 1].x, acc[2 * g + 1].y);
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
#pragma unroll
        for (int g = 0; g < NB / 4; ++g) {
          if (4 * g >= n) break;
          if ((g & 1) == w) {
            const float4 o = cb[g * kTileRows];
            acc[2 * g].x += o.x;
            acc[2 * g].y += o.y;
            acc[2 * g + 1].x += o.z;
            acc[2 * g + 1].y += o.w;
          }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      }
    };
    pdl_wait();  // the activations' scales come from the preparation kernel in front
    if (tid - kConvWarps * 32 < a.batch) xinv[tid - kConvWarps * 32] = __ldg(a.xinv + tid - kConvWarps * 32);
    asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
    for (; wk.live; wk.next_item(a)) {
      const int n = block_cols<NB>(a, wk.nb);
      const int row = (wk.group * TT + t) * kTileRows + r;
      float rs = 1.f, rb = 0.f;
      if (F == Q_FP8 && row < a.out_dim) {
        rs = __ldg(a.scale + row);
        if (a.bias) rb = __ldg(a.bias + row);
      }
      auto store = [&](int j, float v) {  // activation row j of the block
        const int m = wk.nb * NB + j;
        if (m < a.batch && row < a.out_dim) {
          v = (v * T::kUnit) * xinv[m];
          a.out[(size_t)m * a.out_dim + row] = F == Q_FP8 ? fmaf(v, rs, rb) : v;
        }
      };
      if (kItemBlock) {
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(df + 8 * dc.s, dc.ph, a.status, 810));
        if (ok) {
          tc_fence_after();
#pragma unroll 1
          for (int j0 = 0; j0 < n; j0 += 16) {
            uint32_t d[16];
            tmem_ld16(dbase + dc.s * a.dcol + j0, d);
            tmem_wait_ld(d);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              if (a.splits > 1 && wk.tail >= 0) break;
              store(j0 + j, __uint_as_float(d[j]));
            }
          }
          tc_fence_before();
          warp_arrive(de + 8 * dc.s, lane);
        }
        dc.next(DT);
      } else {
#pragma unroll
        for (int j = 0; j < NB / 2; ++j) acc[j] = make_float2(0.f, 0.f);
        // one accumulator block: read, released, added times sc
        auto take = [&](float sc) {
          ok = __all_sync(0xffffffffu, mbar_wait(df + 8 * dc.s, dc.ph, a.status, 812));
          if (!ok) return;
          tc_fence_after();
          if (e == 0) { MARK(5, mk); }
          const float2 sc2 = make_float2(sc, sc);
#pragma unroll
          for (int j0 = 0; j0 < NB; j0 += 32) {
            if (j0 < n) {
              uint32_t d[2][16];
              tmem_ld16(dbase + dc.s * a.dcol + j0, d[0]);
              if (j0 + 16 < n) {  // (a block may have 16 columns, and the last one ends where the allocation does)
                tmem_ld16(dbase + dc.s * a.dcol + j0 + 16, d[1]);
                tmem_wait_ld(d[1]);
              } else {
#pragma unroll
                for (int j = 0; j < 16; ++j) d[1][j] = 0;
              }
              tmem_wait_ld(d[0]);
              if (j0 + 32 >= n) {
                tc_fence_before();
                warp_arrive(de + 8 * dc.s, lane);
              }
#pragma unroll
              for (int j = 0; j < 16; ++j)
                fma2(acc[j0 / 2 + j], sc2, make_float2(__uint_as_float(d[j / 8][(2 * j) & 15]), __uint_as_float(d[j / 8][(2 * j + 1) & 15])));
            }
          }
          dc.next(DT);
          if (e == 0) { MARK(6, mk); }
          TP(++mk;)
        };
        const int chunks = wk.c1 - wk.c;
        if (kLong) {
          for (int ci = 0; ci < chunks && ok; ci += kSeg) take(1.f);
        } else {
          for (int ci = 0; ci < chunks && ok; ++ci) {
            ok = __all_sync(0xffffffffu, mbar_wait(wfull + 8 * wc.s, wc.ph, a.status, 811));
            if (!ok) break;
            const unsigned char* mrow = wring + wc.s * T::kSlot + T::kWBytes + r * (F == Q_Q6K ? 16 : T::kMeta);
            uint4 mv = *reinterpret_cast<const uint4*>(mrow);
            uint32_t m4 = 0;  // Q6_K: d; streaming Q8_0: the fifth pair of scales
            if (F == Q_Q6K && TILED) m4 = *reinterpret_cast<const unsigned short*>(mrow + 2048 - r * 14);
            else if (F == Q_Q6K || (F == Q_Q80 && !TILED)) m4 = *reinterpret_cast<const uint32_t*>(F == Q_Q6K ? mrow + 2048 - r * 12 : mrow + 16);
            // the metadata is in registers (the reduction consumes it): the slot is free for the next load
            if (__reduce_or_sync(0xffffffffu, mv.x | mv.y | mv.z | mv.w | m4 | 1u) && lane == 0) mbar_arrive(wempty + 8 * wc.s);
            wc.next(SW);
            if (TT == 2) wc.next(SW);
            const int c = wk.chunk(wk.c + ci);
            if (F == Q_Q6K && !TILED) m4 >>= 16 * (int)(((size_t)row * a.nchunks + c) & 1);
            if (F == Q_Q80 && !TILED) {
              if (((size_t)row * (a.in_dim / 32)) & 1) {  // the row's scales start in the middle of a pair
                mv = make_uint4(__funnelshift_r(mv.x, mv.y, 16), __funnelshift_r(mv.y, mv.z, 16), __funnelshift_r(mv.z, mv.w, 16),
                                __funnelshift_r(mv.w, m4, 16));
              }
            }
            auto word = [&](int k) { return k == 0 ? mv.x : k == 1 ? mv.y : k == 2 ? mv.z : mv.w; };
#pragma unroll 1
            for (int u = kChunk ? UPC - 1 : 0; u < UPC && ok; ++u) {
              const int b0 = (TT == 2 ? u : w) * kPer;  // the unit's first block in the chunk
#pragma unroll 1
              for (int k = 0; k < kPer && ok; ++k) {
                const int b = b0 + k;
                float sc;
                if (F == Q_MLX4) {
                  sc = __uint_as_float(word(b) << 16);
                } else if (F == Q_Q80) {
                  sc = __half2float(__ushort_as_half((unsigned short)(word(b >> 1) >> (16 * (b & 1)))));
                  if (!TILED && c * 8 + b >= a.in_dim / 32) sc = 0.f;  // past the row: no scale of its own
                } else if (F == Q_Q6K) {
                  const float q = (float)(signed char)((word(b >> 2) >> (8 * (b & 3))) & 0xFFu);
                  sc = __fmul_rn(__half2float(__ushort_as_half((unsigned short)(m4 & 0xFFFFu))), q);  // d * scale, rounded as dequantRowQ6K does
                } else {
                  sc = __half2float(__ushort_as_half((unsigned short)(mv.x & 0xFFFFu)));
                }
                take(sc);
              }
              // the affine term: biases times sums of x, or minus dmin times (minima times sums of x)
              if (T::kAux != 0 && ok && aux_here(w, ci, u))
                take(F == Q_MLX4 ? 1.f : -__half2float(__ushort_as_half((unsigned short)(mv.x >> 16))));
            }
          }
        }
      }
      // ---- the item is complete (every epilogue warp comes through here, waits given up or not) ----
      if (a.splits > 1 && wk.tail >= 0) break;  // the CTA's last item, shared with the cluster: below
      if constexpr (!kItemBlock) {
        combine(n);
        if (ok) {
#pragma unroll
          for (int g = 0; g < NB / 4; ++g) {
            // (with two tiles the way out costs Q5_K and Q6_K registers in the main loop: Q6_K 6144x24832 x91 392 us
            // against 386, where Q8_0 14336x4096 x200 takes 148 with it and 157 without)
            if ((TT == 1 || (F != Q_Q5K && F != Q_Q6K)) && 4 * g >= n) break;
            if (4 * g < n && (TT == 2 || (g & 1) == w)) {
              store(4 * g, acc[2 * g].x);
              store(4 * g + 1, acc[2 * g].y);
              store(4 * g + 2, acc[2 * g + 1].x);
              store(4 * g + 3, acc[2 * g + 1].y);
            }
          }
        }
      }
    }
    if (a.splits > 1) {
      // the sums of the item that the cluster shares go to the CTA's own rings, which are idle once both
      // pipes' blocks have been read: [pipe][group of four columns][row]
      asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
      if (tid == kConvWarps * 32) {
        shared_item[0] = wk.live ? wk.group : -1;
        shared_item[1] = wk.nb;
        shared_item[2] = wk.split;
      }
      float4* ring = reinterpret_cast<float4*>(wring) + (size_t)w * (NB / 4) * kTileRows + r;
      if (wk.live) {
        if constexpr (kItemBlock) {
          // (the block is still in TMEM: nothing has been opened after it)
          tc_fence_after();
#pragma unroll 1
          for (int j0 = 0; j0 < block_cols<NB>(a, wk.nb); j0 += 16) {
            uint32_t d[16];
            tmem_ld16(dbase + j0, d);
            tmem_wait_ld(d);
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              ring[(j0 + j) / 4 * kTileRows] = make_float4(__uint_as_float(d[j]), __uint_as_float(d[j + 1]), __uint_as_float(d[j + 2]), __uint_as_float(d[j + 3]));
          }
        } else {
#pragma unroll
          for (int g = 0; g < NB / 4; ++g) {
            if (4 * g >= block_cols<NB>(a, wk.nb)) break;
            ring[g * kTileRows] = make_float4(acc[2 * g].x, acc[2 * g].y, acc[2 * g + 1].x, acc[2 * g + 1].y);
          }
        }
      }
      if (e == 0) { MARK(7, 2); }
    }
  }
  if (a.splits > 1) {
    // The K splits of the last item are the CTAs of this cluster (rank == split), and each finishes a share of
    // the columns with all of its warps: the others' sums, four columns a load, added in split order (TT = 1:
    // two a split, one from each pipe), and stored.  Everything here runs once, so what it costs is fetching
    // its instructions: short loops, hardly unrolled.  (B200, us a call, with
    // sums pushed to their owners and eight warps at the end: Q4_K 14336x4096 x64 33.8 -> 31.6, MLX4 6144x4096
    // x100 24.8 -> 22.7, bf16 8192x8192 x64 25.6 -> 24.4.)
    __syncwarp();
    cluster_sync_all();
    const int group = shared_item[0], nb = shared_item[1];
    if (warp == 0) { MARK(7, 3); }
    if (group >= 0 && warp < kWarpMMA) {
      constexpr int kPipes = 3 - TT;  // parts of a split's sum
      const int n = block_cols<NB>(a, nb), S = a.splits, sg = ((n + S - 1) / S + 3) / 4, r = tid & (kTileRows - 1);
      const int g0 = shared_item[2] * sg, ng = (g0 + sg < n / 4 ? g0 + sg : n / 4) - g0;
#pragma unroll 1
      for (int u = warp >> 2; u < ng * TT; u += kWarpMMA / 4) {
        const int t = TT == 2 && u >= ng ? 1 : 0, g = g0 + u - t * ng, row = (group * TT + t) * kTileRows + r;
        const uint32_t at = smem_u32(wring) + (uint32_t)((t * (NB / 4) + g) * kTileRows + r) * 16;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
        for (int s0 = 0; s0 < S; s0 += 2 * TT) {
          float4 q[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int s2 = s0 + k / kPipes;
            q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (s2 < S)
              asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(q[k].x), "=f"(q[k].y), "=f"(q[k].z), "=f"(q[k].w)
                           : "r"(cluster_map(at + (k % kPipes) * (NB * kTileRows * 4), s2)) : "memory");
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) v = make_float4(v.x + q[k].x, v.y + q[k].y, v.z + q[k].z, v.w + q[k].w);
        }
        if (row >= a.out_dim) continue;
        const float rs = F == Q_FP8 ? __ldg(a.scale + row) : 1.f, rb = F == Q_FP8 && a.bias ? __ldg(a.bias + row) : 0.f;
        const int m = nb * NB + 4 * g;
        float* o = a.out + (size_t)m * a.out_dim + row;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (m + j < a.batch) {
            const float y = ((j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w) * T::kUnit) * xinv[m + j];
            o[(size_t)j * a.out_dim] = F == Q_FP8 ? fmaf(y, rs, rb) : y;
          }
        }
      }
    }
    __syncwarp();
    if (warp == 0) { MARK(7, 5); }
    // nobody leaves while its sums are being read (they are in registers and added by now: nothing to publish)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    if (warp == 0) { MARK(7, 6); }
  }
  // (the next kernel's CTAs are asked for now and not at the start: the preparation kernel of a following
  // product would crowd onto the few SMs this one leaves free and do all its work there)
  if (warp == kConvWarps) { MARK(7, 1); }
  pdl_launch_dependents();
  // ---- wind down: everyone meets, outstanding copies are drained, TMEM is returned ----
  tc_fence_before();
  __syncthreads();
  if (warp == kWarpB && lane == 0 && *reinterpret_cast<volatile int*>(a.status) != 0) {
    // a waiter gave up: bulk copies may still be in flight; give every slot a bounded chance to land
    for (int s = 0; s < SW + SB; ++s) {
      const uint32_t bar = s < SW ? wfull + 8 * s : bfull + 8 * (s - SW);
      long long t0 = clock64();
      while (!mbar_try_wait(bar, 0) && !mbar_try_wait(bar, 1) && clock64() - t0 < kTimeoutCycles / 8) {
      }
    }
  }
  __syncthreads();
  if (warp == kWarpMMA) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

// ---- host side ---------------------------------------------------------------------------------------

constexpr int kMaxIn = 65536;
constexpr size_t kXbBytes = (size_t)64 << 20;       // prepared activations
constexpr size_t kXauxBytes = (size_t)(kMaxRows / 64) * (kMaxIn / kChunkK) * 64 * 64;
constexpr size_t kFlagBytes = (size_t)(kMaxRows / 64) * (kMaxIn / kChunkK) * 64;
constexpr size_t kSmemBudget2 = 227 * 1024;         // all that a CTA may have

bool carve(QBufs* b, size_t xb_bytes) {
  const size_t total = xb_bytes + kXauxBytes + kMaxRows * 4 + kFlagBytes + 256;
  unsigned char* p = nullptr;
  if (cudaMalloc(&p, total) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  b->xb = p;
  b->xb_bytes = xb_bytes;
  b->xaux = b->xb + xb_bytes;
  b->xinv = reinterpret_cast<float*>(b->xaux + kXauxBytes);
  b->flags = reinterpret_cast<unsigned char*>(b->xinv + kMaxRows);
  b->status = reinterpret_cast<int*>(b->flags + kFlagBytes);
  return true;
}

// The tiled layouts' area, one per device (goph_b200.h asks callers for an order between such calls).
// Allocated on a device's first product of this kind; published only when complete.
QBufs* q_bufs(int device, bool allocate = true) {
  static QBufs bufs[kMaxDevices];
  static bool ready[kMaxDevices] = {};
  static std::mutex mu;
  if (device < 0 || device >= kMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (ready[device]) return &bufs[device];
  if (!allocate || !carve(&bufs[device], kXbBytes)) return nullptr;
  if (cudaMemset(bufs[device].status, 0, 256) != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess) {
    cudaGetLastError();
    cudaFree(bufs[device].xb);
    return nullptr;
  }
  ready[device] = true;
  return &bufs[device];
}

// The other layouts' areas.  The kernels for few rows that also serve these layouts need no scratch, so callers may
// use them on streams without an order between them, from several threads and under capture (the work-list products of every
// layout as well): every stream has an area of its own (found by the stream's id, which no later stream gets again).  Where none is to be had -- under
// capture, since a graph may be replayed beside anything; on the streams after the first kStreamAreas of a device;
// without memory -- the call goes to the kernels for few rows.  Areas go back with the device's last weight.
constexpr int kStreamAreas = 8;
static_assert(kStreamXbBytes == (size_t)64 * kMaxIn * 6, "one block of rows of the widest matrix");

struct StreamAreas {
  std::mutex mu;
  int weights = 0;  // handles of the device
  int n = 0;
  int lost_status = 0;  // of areas given back
  unsigned long long id[kStreamAreas];
  QBufs bufs[kStreamAreas];
};

StreamAreas& stream_areas(int device) {
  static StreamAreas areas[kMaxDevices];
  return areas[device];
}

// Clusters of `size` CTAs that the device holds at once (every CTA takes a whole SM, so this is a
// property of how the SMs are grouped); asked once per device and size.
int cluster_room(int device, int size) {
  static std::mutex mu;
  static int room[kMaxDevices][kMaxSplits + 1];
  static bool known[kMaxDevices][kMaxSplits + 1] = {};
  if (size == 1) return device_state(device).sm_count;
  std::lock_guard<std::mutex> lock(mu);
  if (!known[device][size]) {
    auto kern = qg_kernel<Q_MLX4, true, 1, 64>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget2);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = size;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(size * 16);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBudget2;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    room[device][size] = n;
    known[device][size] = true;
  }
  return room[device][size];
}

// How a launch is cut up: row tiles per item, whole items (a multiple of the grid), the items after
// them and the CTAs that share each of these.
struct Plan {
  int TT, grid, nfull, ntail, splits;
};

// The plan with the smallest estimate, in cycles of the busiest SM (packed formats are counted as a byte a weight, the
// conversion of their bits being what a chunk waits for).  A chunk of an item takes the
// largest of the tensor pipe's time (half a cycle per column and K16 step), the converters' and the
// hand-overs' (tile_cycles) and what the L2 can hand to one SM (45 bytes a cycle); sharing the last items costs two
// meetings of the cluster and the exchange.  max_chunks: longest K range of an item.  The option mlx_splits asks
// for a number of CTAs per shared item, as far as there is a plan with that many.
bool choose_plan(int device, int ntiles, int nchunks, int nblocks, int n, int pieces, int wbytes, double tile_cycles, int NB, int max_chunks, Plan* best) {
  double best_cost = -1;
  int want = options().mlx_splits < kMaxSplits ? options().mlx_splits : kMaxSplits;
  if (want > nchunks) want = nchunks;
  for (int TT = NB == 128 ? 2 : 1; TT <= 2; ++TT) {
    if (TT == 2 && ntiles < 2) break;
    const int items = (ntiles + TT - 1) / TT * nblocks;
    const double mma = TT * 8.0 * pieces * n, conv = tile_cycles * TT, mem = (TT * (double)wbytes + pieces * n * 512.0) / 45;
    const double chunk = mma > conv ? (mma > mem ? mma : mem) : (conv > mem ? conv : mem);
    for (int S = 1; S <= kMaxSplits && S <= nchunks; ++S) {
      if (S > 1 && !options().mlx_cluster) break;
      const int clusters = cluster_room(device, S);
      if (clusters < 1) continue;
      const int grid = clusters * S;
      const int nfull = items / grid * grid, ntail = items - nfull;
      if (ntail > clusters || (S > 1 && ntail == 0)) continue;  // the shared items are the last thing a cluster does
      if ((nfull && nchunks > max_chunks) || (ntail && (nchunks + S - 1) / S > max_chunks)) continue;
      double cost = (nfull / grid * (nchunks * chunk + 1500.0)) + (ntail ? (nchunks + S - 1) / S * chunk + 1500.0 : 0) + (S > 1 ? 1500.0 + TT * n * 8.0 : 0) +
                    (want && S != want ? 1e12 : 0);
      // Clusters of three, five or seven that the device only just holds do not start all at once behind another kernel, and one that starts late is late for all
      // its items (B200, us a call: Q8_0 3250x14080 x29, 26 clusters of five 46.7, of four 33.1; Q4_K 28672x8192 x256, 45 of three 432, of two 289).  Those of four and six do: Q4_K
      // 19072x8192 x9, 132 whole items and 17 shared by six 49.8, two tiles an item by one CTA each 62.1; 10000x4096 x200 by four 58.3, by two 65.8.
      if (S > 2 && S % 2 && (nfull ? grid / S : ntail) == clusters) cost *= 1.35;
      if (best_cost < 0 || cost < best_cost) {
        best_cost = cost;
        *best = Plan{TT, nfull ? grid : ntail * S, nfull, ntail, S};
      }
    }
  }
  return best_cost >= 0;
}

// What a chunk of one tile costs where its conversion and the hand-overs of its accumulator blocks set the pace (28672x4096, 16 and 64 rows).  With
// 300 for every format the plan took two tiles an item, and fewer items than SMs, where one was better (B200, us a call): Q8_0 6000x2048 x200 43.4 ->
// 36.5, 12000x1024 x30 14.6 -> 12.8, 1500x12288 x100 40.5 -> 37.4, Q6_K 20000x1024 x64 39.1 -> 29.7, 2000x8192 x40 39.9 -> 31.4.  The others keep it: what
// two tiles of an item share, the B tiles, counts for more than the estimate has (Q4_K 14336x4096 x64 29.7, with one tile 35.6, 3584x18944 x11 28.0
// and 30.4; Q5_K 28.0 and 32.1); MLX with foldable scales and FP8 close a block in 16 chunks and wait for the L2 or the tensor cores.
template <int F>
double tile_cycles(int n) {
  const double more = (n - 16) / 48.0;  // of 64 columns
  if (F == Q_Q80) return 3100 + 1500 * more;
  if (F == Q_Q6K) return 5500 + 2100 * more;
  return 300;
}

template <int F, bool TILED, int TT, int NB>
int launch_product(QArgs& a, const QMapArgs<TILED>& maps, const Plan& p, int n, int device, cudaStream_t stream) {
  typedef QF<F, TILED> T;
  // B slots hold every piece of half a chunk and the affine term's sums: two at least, more where they are
  // small; the weight ring gets the rest
  a.bslot = n * 256 * a.pmax + T::kAux * n * 32;
  a.comb = TT == 1 ? n * kTileRows * 4 : 0;
  a.bslots = (int)((size_t)(NB == 128 ? 96 : 104) * 1024 / a.bslot);
  if (a.bslots > 4) a.bslots = 4;  // (six: FP8 8192x28672 x5 53.2 us, four 49.4, two 54.7: small B slots leave the room to the weights)
  // A pipe must see every round of the slots that it waits for (a parity wait cannot tell a round from the
  // one two before it): where the pipes take turns, their slots stay apart by an even depth.
  if (TT == 1) a.bslots &= ~1;
  a.dcol = n <= 16 ? 16 : n <= 32 ? 32 : NB;
  const size_t fixed = 1024 + 2048 + (size_t)a.bslots * a.bslot + a.comb + (T::kAux ? (T::kLong && NB == 64 ? 6 : 4) * 4096 : 0);
  a.wslots = (int)((kSmemBudget2 - fixed) / T::kSlot);
  if (a.wslots > 10) a.wslots = 10;
  a.wslots &= ~1;  // (the same for the tiles of an item, or the converter groups of a pipe)
  if (a.wslots < 2 || a.bslots < 2) return fail(GOPH_E_UNSUPPORTED, "several-row products: no room for the rings");
  size_t smem = fixed + (size_t)a.wslots * T::kSlot;
  if (smem < 120 * 1024) smem = 120 * 1024;  // one CTA per SM (the kernel owns all of TMEM)
  auto kern = qg_kernel<F, TILED, TT, NB>;
  static bool sized[kMaxDevices] = {};
  if (!sized[device]) {
    GOPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget2));
    sized[device] = true;
  }
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = p.splits > 1 ? 2 : 1;
  cfg.gridDim = dim3(p.grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  note_launch();
  GOPH_CUDA(cudaLaunchKernelEx(&cfg, kern, a, maps));
  return GOPH_OK;
}

// What an area of scratch holds of the call's x, so that weights of one call share its preparation.
struct Prepared {
  bool valid = false;
  int order, sums, nb;
  float unit;
};

template <int F, bool TILED, bool XBF16>
int run_rows(const QWeight& w, float* out, const void* x, int batch, QBufs* bufs, Prepared* prep, cudaStream_t stream) {
  typedef QF<F, TILED> T;
  constexpr int pmax = XBF16 ? 1 : 3;
  const int nchunks = (w.in_dim + kChunkK - 1) / kChunkK;
  const size_t xstride = (size_t)w.in_dim * (XBF16 ? 2 : 4);
  for (int b0 = 0; b0 < batch;) {
    // wide column blocks halve the weight traffic where one is read out once per item
    int NB = F == Q_FP8 && TILED && XBF16 && batch - b0 > 64 ? 128 : 64;
    Plan p;
    if (NB == 128) {
      const int rows = batch - b0 < kMaxRows ? batch - b0 : kMaxRows;
      if (!choose_plan(w.device, (w.out_dim + kTileRows - 1) / kTileRows, nchunks, (rows + 127) / 128, rows < 128 ? (rows + 15) & ~15 : 128, 1, T::kSlot, 300, NB, 32, &p))
        NB = 64;
    }
    const size_t block_bytes = (size_t)NB * nchunks * kChunkK * 2 * pmax;
    int cap = (int)(bufs->xb_bytes / block_bytes) * NB;
    if (cap > kMaxRows) cap = kMaxRows;
    const int rows = batch - b0 < cap ? batch - b0 : cap;
    QArgs a;
    memset(&a, 0, sizeof a);
    QMapArgs<TILED> maps;
    if constexpr (!TILED) {
      memcpy(maps.map, w.maps->map, sizeof maps.map);
    }
    a.w = static_cast<const unsigned char*>(w.w);
    a.aux = w.aux;
    a.xb = bufs->xb;
    a.xaux = bufs->xaux;
    a.xinv = bufs->xinv;
    a.flags = XBF16 ? nullptr : bufs->flags;
    a.scale = w.scale;
    a.bias = w.bias;
    a.out = out + (size_t)b0 * w.out_dim;
    a.status = bufs->status;
    a.xb_stride = block_bytes;
    a.out_dim = w.out_dim;
    a.in_dim = w.in_dim;
    a.batch = rows;
    a.ntiles = (w.out_dim + kTileRows - 1) / kTileRows;
    a.nchunks = nchunks;
    a.nblocks = (rows + NB - 1) / NB;
    a.pmax = pmax;
    const int n = rows >= NB ? NB : (rows + 15) & ~15;  // columns of the first (widest) block
    if (!choose_plan(w.device, a.ntiles, nchunks, a.nblocks, n, T::kMLX ? 1 : pmax, T::kPacked ? kTileRows * 288 : T::kSlot, tile_cycles<F>(n), NB, NB == 128 ? 32 : 1 << 20, &p))
      return fail(GOPH_E_UNSUPPORTED, "several-row products: the device holds no CTA of this kernel");
    a.nfull = p.nfull;
    a.ntail = p.ntail;
    a.splits = p.splits;

    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    // two CTAs per SM where the row has the chunks for it (a warp takes one)
    int slices = 2 * device_state(w.device).sm_count / rows;
    if (slices > (nchunks + 7) / 8) slices = (nchunks + 7) / 8;
    cfg.gridDim = dim3(rows, slices < 1 ? 1 : slices);
    cfg.blockDim = dim3(kPrepThreads);
    if (!(prep->valid && rows == batch && prep->order == T::kOrder && prep->sums == T::kSums && prep->nb == NB && prep->unit == T::kUnit)) {
      note_launch();
      GOPH_CUDA(cudaLaunchKernelEx(&cfg, qg_prep_x_kernel<T::kOrder, T::kSums, XBF16>,
                                   static_cast<const void*>(static_cast<const unsigned char*>(x) + (size_t)b0 * xstride), bufs->xb,
                                   bufs->xaux, bufs->xinv, bufs->flags, rows, w.in_dim, nchunks, NB, a.xb_stride, 1.f / T::kUnit));
      prep->valid = rows == batch;
      prep->order = T::kOrder;
      prep->sums = T::kSums;
      prep->nb = NB;
      prep->unit = T::kUnit;
    }
    int rc;
    if constexpr (F == Q_FP8 && TILED && XBF16) {
      if (NB == 128) rc = launch_product<F, TILED, 2, 128>(a, maps, p, n, w.device, stream);
      else rc = p.TT == 2 ? launch_product<F, TILED, 2, 64>(a, maps, p, n, w.device, stream) : launch_product<F, TILED, 1, 64>(a, maps, p, n, w.device, stream);
    } else {
      rc = p.TT == 2 ? launch_product<F, TILED, 2, 64>(a, maps, p, n, w.device, stream) : launch_product<F, TILED, 1, 64>(a, maps, p, n, w.device, stream);
    }
    if (rc) return rc;
    b0 += rows;
  }
  return GOPH_OK;
}

template <int F>
int run_fmt(const QWeight& w, float* out, const void* x, bool x_bf16, int batch, QBufs* bufs, Prepared* prep, cudaStream_t stream) {
  if constexpr (F == Q_MLX4 || F == Q_MLX4F || F == Q_FP8) {
    if (x_bf16)
      return w.tiled ? run_rows<F, true, true>(w, out, x, batch, bufs, prep, stream) : fail(GOPH_E_UNSUPPORTED, "bf16 activations need the tiled layout");
  } else if (x_bf16) {
    return fail(GOPH_E_UNSUPPORTED, "bf16 activations: MLX 4-bit and FP8 only");
  }
  return w.tiled ? run_rows<F, true, false>(w, out, x, batch, bufs, prep, stream) : run_rows<F, false, false>(w, out, x, batch, bufs, prep, stream);
}

int run_one(const QWeight& w, float* out, const void* x, bool x_bf16, int batch, QBufs* bufs, Prepared* prep, cudaStream_t stream) {
  switch (w.fmt) {
    case Q_MLX4: return run_fmt<Q_MLX4>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_MLX4F: return run_fmt<Q_MLX4F>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_Q4K: return run_fmt<Q_Q4K>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_Q5K: return run_fmt<Q_Q5K>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_Q6K: return run_fmt<Q_Q6K>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_Q80: return run_fmt<Q_Q80>(w, out, x, x_bf16, batch, bufs, prep, stream);
    case Q_FP8: return run_fmt<Q_FP8>(w, out, x, x_bf16, batch, bufs, prep, stream);
  }
  return fail(GOPH_E_INVALID, "unknown weight format %d", w.fmt);
}

}  // namespace

// The lines lie where this kernel's time and the few-row kernels' met (B200, us a call: few-row / this).
// Tiled layouts: the few-row kernel takes 8 rows a launch, and its time grows with the rows; it is bound by its instructions from
// four rows on, sooner where scales are packed.  Q6_K and Q8_0, with a block per 16 or 32 elements here too, gain later.
// Other layouts: MLX rows up to the line are on the integer tensor cores too.  GGUF matrices have these layouts only below 0.5 Mi weights (Q6_K 1.5 Mi) or 256
// rows, or by option; the lines beyond are for the option, and hold small tiled matrices on exact sums (gguf.cu).  The CUDA-core
// kernels' time grows with the rows and the weights (four rows a pass, eight in two), this
// one's hardly, but two launches and the start cost it 7 to 9 us (Q6_K, a block per 16 elements, 9 to 19).  For Q8_0
// the lines are where the times meet.  Elsewhere this kernel's f32 sums in tensor memory are
// a little coarser than those of the CUDA cores (against 64 bits, 4096 elements a row: Q4_K 4.6e-7 / 2.9e-7, Q5_K 4.5e-7 /
// 2.9e-7, Q6_K 1.3e-7 / 1.0e-7, MLX4 1.4e-6 / 4.8e-7, FP8 1.5e-6 / 1.0e-7; but Q8_0 1.7e-7 / 4.4e-7), and the lines stay above the
// rows from which it is the faster one.  (MLX rows of up to 2048 elements: 2048x1024 4.9e-7 / 5.1e-7, but where no K range is cut 28672x1088 2.7e-6 /
// 5.4e-7, and with x of bf16 values 1.2e-7 / 0.8e-7 and 1.0e-6 / 0.9e-7.)  A weight of `weights` that share x
// costs a launch of its own here, while the MLX streaming kernel takes all of them in one; out_dim is their sum.
bool qgemm_wants(int fmt, bool tiled, bool x_bf16, long out_dim, int in_dim, int batch, int weights) {
  if (x_bf16) return fmt != Q_FP8 || batch > 16;  // FP8 14336x4096: 16 rows 16.7 / 18.2, 24 rows 22.7 / 21.2
  const long size = out_dim * in_dim, Mi = 1l << 20;
  if (tiled) {
    switch (fmt) {
      case Q_FP8: return batch > 4;  // 4096x14336 4 rows 17.4 / 19.7, 5 rows 34.1 / 19.8
      // 18944 rows: a tile for each of 148 SMs.  MLX 8 rows 4096x4096 8.5 / 10.7, 14336x4096 16.0 / 21.4, 18688x4096 16.5 / 25.1, 19072x4096 26.7 / 26.4, 28672x8192 50.9 / 47.1
      case Q_MLX4: case Q_MLX4F: return batch > (out_dim <= 18944 ? 8 : 4);
      // 9472: two.  Q4_K 4 rows 14336x4096 14.0 / 21.3; 8 rows 4096x4096 10.1 / 11.6, 4096x14336 21.2 / 24.4, 8192x8192 23.6 / 22.9, 14336x4096 21.6 / 21.3
      case Q_Q4K: case Q_Q5K: return batch > (out_dim <= 9472 && size < 64 * Mi ? 8 : 4);
      // 4096x4096 10 rows 18.2 / 19.2, 12 rows 19.9 / 19.3; 14336x4096 12 rows 46.8 / 53.6, 16 rows 53.1 / 53.7
      case Q_Q6K: return batch > (size <= 16 * Mi ? 10 : 12);
      default: return batch > (size <= 16 * Mi ? 8 : 12);  // Q8_0 4096x4096 9 rows 14.1 / 13.8; 14336x4096 12 rows 29.1 / 33.5, 16 rows 34.8 / 33.6
    }
  }
  if (weights > 1) {  // (MLX) by their mean size: 2048, 1024 and 1024 rows of 1024 at 16 rows 21.4 / 20.2, at 20 28.2 / 22.3;
    const long mean = size / weights;  // 2048, 512, 512 of 2048 at 9 21.6 / 22.6, at 12 24.9 / 22.7; twice 2048x2048 at 8 18.1 / 16.4;
    // four of 1024x4096 at 8 19.4 / 38.7 (and 1.6e-7 / 7.7e-7 off)
    return batch > (mean < Mi ? 24 : mean < 2 * Mi ? 16 : mean < 3 * Mi ? 10 : mean < 5 * Mi || size <= 12 * Mi ? 8 : 4);
  }
  // Above 8 Mi weights this layout is the exception (widths that no tile takes, NaN codes, the layout options).
  // in_dim above 8192: of x the CUDA-core kernels' shared memory holds four rows (Q8_0, FP8) for one CTA an SM only, or two.
  const bool small = size < 4 * Mi, long_rows = size >= 6 * Mi && in_dim >= 4096, wide_x = in_dim > 8192;
  switch (fmt) {
    case Q_Q6K:  // 1024x1024 16 rows 10.7 / 9.3; 3072x1024 4 rows 5.6 / 9.6, 9 rows 12.7 / 9.6; 2048x2048 8 rows 11.7 / 13.8, 9 rows 15.3 / 13.8; 1536x4096
                 // 4 rows 11.5 / 13.5, 5 rows 17.8 / 13.5; 28672x4096 8 rows 97 / 107, 9 rows 148 / 107; 8192x8192 4 rows 57 / 57
      return batch > (size < 2 * Mi ? 24 : wide_x && size >= 8 * Mi ? 8 : size > 16 * Mi ? 24 : long_rows ? 12 : 16);
    case Q_Q5K:  // 512x2048 8 rows 8.1 / 8.3, 9 rows 11.0 / 8.3; 2048x2048 4 rows 7.4 / 9.3, 5 rows 12.7 / 9.3; 1536x4096 2 rows 8.6 / 9.7, 3 rows 12.6 / 9.7
      return batch > (size < 2 * Mi ? 10 : long_rows || size >= 8 * Mi ? 4 : 8);
    case Q_Q80: {  // 1024x2048 8 rows 8.0 / 9.1, 9 rows 10.8 / 9.1; 3072x1024 4 rows 5.4 / 8.5, 5 rows 9.1 / 8.5; 2048x2048 6.6 / 10.7, 11.1 / 10.7;
      // 1024x7168 13.2 / 14.9, 21.6 / 14.9; short rows, and very many, fill the SMs with four rows: 12000x1056 12.9 / 14.0, 22.0 / 14.0; 19072x1024 12.8 / 19.3,
      // 23.7 / 19.4; 14336x4128 39.1 / 39.8, 74.9 / 39.8; 28672x4160 68.2 / 68.3, 133 / 68; longer ones with two, and very many whose last 512 elements (a
      // warp's step) are not full: 5000x2080 2 rows 10.0 / 12.7, 3 rows 15.6 / 12.7; 4096x4160 14.2 / 18.3, 22.2 / 18.4; 8192x6240 30.8 / 32.9, 74.7 / 33.0;
      // 512x14336 20.8 / 20.9, 36.3 / 20.8; 28672x1056 17.3 / 23.3, 24.1 / 23.3; 65536x544 23.2 / 28.2, 34.6 / 28.1
      const bool many = in_dim % 512 != 0 && out_dim * ((in_dim + 511) / 512 * 512) > 40 * Mi;
      const bool two = wide_x || (size >= 8 * Mi && (in_dim >= 6144 || (in_dim >= 2048 ? size < 48 * Mi : many)));
      return batch > (2 * size < 5 * Mi ? 8 : two ? 2 : 4);
    }
    case Q_MLX4: case Q_MLX4F: return batch > (size <= 5 * Mi ? 8 : 4);  // 8 rows 2048x2048 6.9 / 8.6, 512x8192 9.9 / 11.3, 5722x1280 11.9 / 8.8, 8192x2112 12.0 / 11.8
    case Q_Q4K:
      // 1536x4096 2 rows 7.7 / 9.4, 3 rows 12.2 / 9.4
      return batch > (small ? 8 : (long_rows || (size >= 8 * Mi && in_dim > 1024)) && size <= 64 * Mi ? 2 : 4);
    default:     // FP8 1024x1024 8 rows 5.3 / 7.0, 9 rows 7.1 / 7.0; 2048x2048 4 rows 5.7 / 8.2, 5 rows 9.4 / 8.1; 4096x4160 2 rows 11.4 / 10.1; 512x14336
                 // 2 rows 12.7 / 13.4, 3 rows 22.7 / 13.4; 8192x8256 2 rows 36.2 / 15.8
      return batch > (small ? 8 : wide_x ? 2 : size >= 16 * Mi && size < 48 * Mi ? 3 : 4);
  }
}

// Tensor map of `rows` rows of `bytes` bytes, `pitch` apart: boxes of 128 rows and `box` bytes, zeros past the edges.
static bool encode_map(CUtensorMap* map, const void* base, uint64_t bytes, uint64_t rows, uint64_t pitch, int box) {
  typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<Encode>(f);
  }();
  if (!encode) return false;
  const cuuint64_t dims[2] = {bytes, rows}, pitches[1] = {pitch};
  const cuuint32_t boxes[2] = {(cuuint32_t)box, kTileRows}, steps[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, pitches, boxes, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                box == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

void qgemm_maps(int fmt, const void* w, const void* aux, int out_dim, int in_dim, QMaps* maps) {
  const uint64_t rows = out_dim, in = in_dim, chunks = in / 256, n = rows * in;
  const unsigned char* hi = static_cast<const unsigned char*>(aux);
  bool ok = true;
  memset(maps, 0, sizeof *maps);
  switch (fmt) {
    case Q_MLX4: case Q_MLX4F:
      ok = encode_map(&maps->map[0], w, in / 2, rows, in / 2, 128) && encode_map(&maps->map[1], aux, (in + 255) / 256 * 16, rows, (in + 255) / 256 * 16, 16);
      break;
    case Q_Q4K: case Q_Q5K: {
      const uint64_t row = chunks * (fmt == Q_Q4K ? 144 : 176);
      ok = encode_map(&maps->map[0], w, row, rows, row, 128) && encode_map(&maps->map[1], w, row, rows, row, 16);
      break;
    }
    case Q_Q6K:
      ok = encode_map(&maps->map[0], w, in / 2, rows, in / 2, 128) && encode_map(&maps->map[1], hi, in / 4, rows, in / 4, 16) &&
           encode_map(&maps->map[2], hi + n / 4, in / 16, rows, in / 16, 16);
      break;
    default:
      ok = in % 16 == 0 && encode_map(&maps->map[0], w, in, rows, in, 128);
  }
  maps->ok = ok;
}

int qgemm(int n, const QWeight* w, float* const* out, const void* x, bool x_bf16, int batch, QBufs* rows, cudaStream_t stream) {
  if ((uintptr_t)x % 16) return fail(GOPH_E_INVALID, "x must be 16-byte aligned");
  bool any[2] = {};
  for (int i = 0; i < n; ++i) {
    if (w[i].in_dim > kMaxIn) return fail(GOPH_E_UNSUPPORTED, "several-row products: in_dim=%d is above %d", w[i].in_dim, kMaxIn);
    any[w[i].tiled && !w[i].unordered] = true;
  }
  // the device's area for tiled weights, the stream's for the others; both are held to the call's last launch
  QBufs* bufs[2] = {any[0] ? rows : nullptr, any[1] ? q_bufs(w[0].device) : nullptr};
  std::unique_lock<std::mutex> held[2];
  Prepared prep[2];
  for (int t = 0; t < 2; ++t) {
    if (!any[t]) continue;
    if (!bufs[t]) return fail(GOPH_E_NOMEM, "cannot allocate the several-row products' device scratch");
    held[t] = std::unique_lock<std::mutex>(bufs[t]->enqueue);
  }
  for (int i = 0; i < n; ++i)
    if (int rc = run_one(w[i], out[i], x, x_bf16, batch, bufs[w[i].tiled && !w[i].unordered], &prep[w[i].tiled && !w[i].unordered], stream)) return rc;
  return GOPH_OK;
}

QBufs* qgemm_scratch(int device, cudaStream_t stream) {
  unsigned long long id = ~0ull;  // the legacy default stream, which is never captured: no questions (0.5 us a call)
  if (stream != nullptr && stream != cudaStreamLegacy) {
    cudaStreamCaptureStatus capture;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone || cudaStreamGetId(stream, &id) != cudaSuccess) {
      cudaGetLastError();
      return nullptr;
    }
  }
  StreamAreas& s = stream_areas(device);
  std::lock_guard<std::mutex> lock(s.mu);
  for (int i = 0; i < s.n; ++i)
    if (s.id[i] == id) return &s.bufs[i];
  if (s.n == kStreamAreas) return nullptr;
  // (another thread may be capturing a stream of its own, which an allocation must not disturb)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  QBufs& b = s.bufs[s.n];
  bool ok = carve(&b, kStreamXbBytes);
  if (ok && cudaMemsetAsync(b.status, 0, 256, stream) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(b.xb);
    ok = false;
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  if (!ok) return nullptr;
  s.id[s.n++] = id;
  return &b;
}

QScratch qgemm_scratch_area(QBufs* b) { return QScratch{b->xb, b->status, &b->enqueue}; }

void qgemm_weights(int device, int change) {
  StreamAreas& s = stream_areas(device);
  std::lock_guard<std::mutex> lock(s.mu);
  s.weights += change;
  if (s.weights > 0) return;
  for (; s.n > 0; --s.n) {  // (reading the status word and freeing both wait for the device)
    QBufs& b = s.bufs[s.n - 1];
    int v = 0;
    if (cudaMemcpy(&v, b.status, sizeof v, cudaMemcpyDeviceToHost) == cudaSuccess && s.lost_status == 0) s.lost_status = v;
    cudaFree(b.xb);
  }
  cudaGetLastError();
}

int qgemm_status(int device) {
  int v = 0;
  if (QBufs* b = q_bufs(device, false)) {
    v = -1;
    cudaMemcpy(&v, b->status, sizeof v, cudaMemcpyDeviceToHost);
  }
  StreamAreas& s = stream_areas(device);
  std::lock_guard<std::mutex> lock(s.mu);
  if (v == 0) v = s.lost_status;
  for (int i = 0; i < s.n && v == 0; ++i) {
    v = -1;
    cudaMemcpy(&v, s.bufs[i].status, sizeof v, cudaMemcpyDeviceToHost);
  }
  return v;
}

void qgemm_status_clear(int device) {
  if (QBufs* b = q_bufs(device, false)) cudaMemset(b->status, 0, sizeof(int));
  StreamAreas& s = stream_areas(device);
  std::lock_guard<std::mutex> lock(s.mu);
  s.lost_status = 0;
  for (int i = 0; i < s.n; ++i) cudaMemset(s.bufs[i].status, 0, sizeof(int));
}

}  // namespace goph

#ifdef GOPH_TUNING
GOPH_API int goph_tuning_probe_q(long long* out512) {
  return cudaMemcpyFromSymbol(out512, goph::g_qg_trace, 8 * 64 * sizeof(long long)) == cudaSuccess ? 0 : -1;
}
#endif
