// Products of up to eight activation rows (FP8: four) with weights in the tiled layouts and row-major MLX and FP8 ones, in exact
// integer arithmetic (FP8: e4m3 pieces, f32) on the tensor cores' register path (mma.sync).
//
// Why this path: at B200's HBM rate one SM has to take in 41 nibbles a clock.  Turned into floats on the CUDA cores a nibble
// costs five to seven lane instructions and an SM has 128 a clock.  Here nibbles stay integers: three logic instructions turn
// a packed word into eight bytes, which are the A fragment of an MMA as they stand; the MMA is exact, and per group of weights
// a scale is applied.  MMAs of 16 x 8 x 32 bytes issue every two clocks on an SM (measured): 256 weights a clock for two
// activation rows, five times what HBM delivers, so there is nothing to gain from tcgen05's rate, which wants the bytes written to
// tensor memory by converter warps and the sums read back by others.  That form, which stood here, handed every 18 KB from
// warp to warp four times, took a whole SM a CTA and got 34 weights a clock; a warp that does it all for its rows got 46 (one row, Q4_K 128256x4096).
//
// Arithmetic
//   * A operand (weights): nibble n as the unsigned byte n, byte formats as they lie in the tile.
//   * B operand (activations): each group of 64 (MLX) or 32 elements of an activation row is put on a common
//     power-of-two scale 2^(E-26), E the exponent of the group's largest magnitude, and every
//     element becomes the integer q = round(x * 2^(26-E)), |q| <= 2^26 -- at least as fine as
//     the f32 spacing of the group's largest elements.  q is written as four balanced base-128
//     digits, one column of signed bytes per digit (with three, an option for bf16-valued x, the fourth is zero).
//   * One accumulator tile per block of weights with a common scale (64, 32 or, Q6_K, 16 elements), exact.  A lane has the sums
//     of two neighbouring digits, d0 + 128 d1, which is a float exactly (Q8_0: rounded once), times 2^(E-26) (or 2^(E-12)),
//     times the block's scale, added in f32; biases or minima times the group's sum of x are added behind it (mlx.GemvTo,
//     backends/mlx/gemv.go:178-209; loader/gguf/quant_matrix.go:281-426).  The lanes of a quad meet when an item ends.
//
// A CTA: eight warps that compute and one that loads.  A stage is 256 elements of a 128-row tile, one bulk copy (the tiled
// layouts store exactly the image of a stage) into a ring guarded by full/empty mbarriers; a warp takes its 16 or 32 rows of a
// stage from ldmatrix to running sums with nobody else.  The activations' digits are made by the CTA itself for its K range
// while the first stages are on their way, or by a launch in front (see launch_one).  Two CTAs share an SM, or one launch's
// CTAs and the next one's, whose first stages are then in shared memory before this launch has ended; products that are over
// in a few stages take an SM each.  Where K is cut, the CTAs of a tile are a cluster and add their sums through its
// first CTA's shared memory (or through scratch), in split order whoever is first.
// Every mbarrier wait is bounded (~2 s): a waiter that gives up records a code in the status word and the CTA winds down.
//
// Measured (B200, us a call among others, weights from HBM; before: the tcgen05 form, five to eight rows of MLX and Q4_K and four of Q4_K the
// f16 kernel of qgemm.cu):
//   one row     MLX4 4096x4096 5.9 -> 4.8, 14336x4096 9.3 -> 7.1, 28672x8192 28.9 -> 23.3; Q4_K 4096x14336 11.1 -> 9.3; Q8_0 28672x8192 43.5 -> 39.7
//   two rows    MLX4 28672x4096 17.8 -> 12.7, Q8_0 4096x4096 7.1 -> 5.4; four: Q4_K 14336x4096 20.9 -> 13.7, Q6_K 28672x8192 80.3 -> 62.1
//   eight rows  MLX4 14336x4096 20.9 -> 15.6, Q8_0 28672x8192 101 -> 54, Q6_K 14336x4096 46.4 -> 27.2
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "goph_internal.cuh"
#include "mlx_mma.cuh"
#include "tc_common.cuh"

namespace goph {

using namespace tc;

constexpr int kTileRows = 128;
constexpr int kChunkK = 256;  // elements of a pipeline stage

// What differs between the weight formats.  A stage is 128 rows x 256 elements, then 16 bytes of scale data per row.
//   MLX4  128 B of nibbles per row (16-byte units XOR-swizzled by row); {scale,bias} bf16 pairs of the 4 groups of 64.
//   Q4K   the same nibble image (one 256-element super-block per row and stage); f16 d, f16 dmin and
//         8 x 12 bits (sc | m << 6), one per 32-element sub-block.
//   Q80   256 signed bytes per row, stored as 8x16-byte matrices [K step][K half][row group][row][16 B]; 8 f16 block scales.
//   Q5K   the nibble image, in which word t of a unit (32 elements) holds elements 4 t .. 4 t + 3 in the low nibbles of its bytes and
//         16 + 4 t .. in the high ones; then the fifth bits: [4 units][row][word t], byte b of which has, from bit 0, those of unit 0 low and
//         high, unit 1 low, ... of byte b; the Q4_K header {d, dmin, 8 x (sc | m << 6)}.
//   Q6K   the same image; two bits beside every nibble: [2 units][row][word t], byte b: unit 0 low, high, unit 1 low, high (the A byte
//         is nibble and bits at its top, the highest one inverted: 4 (q - 32), signed); 16 int8 scales per row, one per 16
//         elements; then f16 d [row].
//   FP8   256 e4m3 bytes per row, in Q80's order; no scales (one per row, applied at the end).  Row-major: two images of 128 rows x 128
//         bytes, 16-byte units XOR-swizzled by row.
//   (Q5K and Q6K are as large as in the file.  Written out to bytes, 1.06 and 1.13 a weight, they were bound by HBM at 1.5 and 1.4 times the time.)
enum { FMT_MLX4 = 0, FMT_Q4K = 1, FMT_Q80 = 2, FMT_Q5K = 3, FMT_Q6K = 4, FMT_FP8 = 5 };
template <int FMT>
struct Fmt {
  static constexpr bool kNibble = FMT != FMT_Q80 && FMT != FMT_FP8;   // a nibble image
  static constexpr bool kWords = FMT == FMT_MLX4 || FMT == FMT_Q4K;   // whose words hold eight consecutive elements
  static constexpr bool kSigned = FMT == FMT_Q80 || FMT == FMT_Q6K;  // A bytes
  static constexpr bool kSums = FMT == FMT_MLX4 || FMT == FMT_Q4K || FMT == FMT_Q5K;  // biases or minima meet the groups' sums of x
  static constexpr int kGroup = FMT == FMT_FP8 ? 256 : FMT == FMT_MLX4 ? 64 : 32;  // elements of an entry of the activation tables
  static constexpr int kGroups = kChunkK / kGroup;
  static constexpr int kHigh = FMT == FMT_Q5K ? 4096 : FMT == FMT_Q6K ? 8192 : 0;  // bits beside the nibbles
  static constexpr int kHighOff = kTileRows * 128;
  static constexpr int kStageWBytes = kTileRows * (kNibble ? 128 : 256) + kHigh;
  static constexpr int kMetaRow = FMT == FMT_FP8 ? 0 : 16;                          // bytes of scales per row and stage
  static constexpr int kDOff = kStageWBytes + kTileRows * kMetaRow;                 // Q6_K: d
  static constexpr int kStageBytes = kDOff + (FMT == FMT_Q6K ? kTileRows * 2 : 0);
};

// Prepared activations of a chunk and up to MB rows: B fragments, then tables.
//   fragments  [pair of K steps][n tile][lane][K step of the pair] x 8 bytes: what mma.m16n8k32 wants of lane 4 n + t (column
//              n = 4 * row + digit).  One row would leave columns 4 to 7 idle: blocks of weights with a scale of their own go in pairs,
//              the digits of the first one's elements stand in columns 0 to 3, of the second one's in 4 to 7, zeros elsewhere, so
//              that one accumulator tile holds both sums (MLX: groups, Q6_K: the halves of a K step, others: K steps).
//   tables     per row, parity p of the lane (even lanes hold the sums of the two low digits, odd ones of the two high ones) and
//              group: the group's scale 2^(E-26) (p = 1: times 2^14) and, where biases or minima want it, its sum of x (p = 0: zero).
//              One row: per p, half of the quad (lanes 0 and 1 finish the pairs' first blocks) and pair (Q6_K: per p and group).
template <int FMT, int MB>
struct XBlock {
  typedef Fmt<FMT> F;
  static constexpr bool kRowTile = FMT == FMT_FP8;  // a tile of columns per activation row, which has six pieces
  static constexpr int NT = kRowTile ? MB : MB == 1 ? 1 : MB / 2;  // n tiles of eight columns
  static constexpr int kFrag = NT * 2048;
  static constexpr int kEntry = F::kSums ? 2 : 1;  // floats
  static constexpr int kTab = FMT == FMT_FP8 ? MB * 4 : MB * 2 * F::kGroups * kEntry;
  static constexpr int kBytes = kFrag + kTab * 4;
  static __host__ __device__ __forceinline__ int frag(int step, int n, int t) {
    return ((step >> 1) * NT + (n >> 3)) * 512 + ((n & 7) * 4 + t) * 16 + (step & 1) * 8;
  }
  static __host__ __device__ __forceinline__ int entry(int m, int p, int g) {
    if (MB == 1 && FMT != FMT_Q6K) return ((p * 2 + (g & 1)) * (F::kGroups / 2) + (g >> 1)) * kEntry;
    return ((m * 2 + p) * F::kGroups + g) * kEntry;
  }
};

__device__ __forceinline__ float f16_lo(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
__device__ __forceinline__ float f16_hi(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }
__device__ __forceinline__ float max_nan(float a, float b) {  // (fmaxf passes over a NaN)
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}

// 2^(field - 127), field > -23: below 1 a subnormal float, which is a power of two exactly as well.
__device__ __forceinline__ float pow2_biased(int field) { return __uint_as_float(field > 0 ? (uint32_t)field << 23 : 1u << (22 + field)); }
// A warp turns the 256 elements of one chunk of activation row m, eight consecutive ones per lane (SPLIT 4: a block of
// four warps, four lanes to the same eight elements, each of which writes one digit), into the row's part of an XBlock.
// The digits come from one sum: q + 64 (1 + 128 + 128^2) has d_j + 64 in its j-th seven bits (the top digit has what is
// left), and a byte pattern d + 64 of seven bits becomes the signed byte.
// The smallest unit is 2^-149: activations keep their bits down to the subnormal floats (their groups' scales are subnormal then).
// A group with a NaN or an infinity has the scale NaN, which is what every product with it becomes (an integer has neither).
// R: chunks at once, each with its own values, place and row (their chains of shuffles interleave).
template <int FMT, int MB, int SPLIT = 1, int R = 1>
__device__ __forceinline__ void prep_chunks(const float (&v)[R][8], int lane, unsigned char* const (&xb)[R], const int (&m)[R], int digits) {
  typedef Fmt<FMT> F;
  typedef XBlock<FMT, MB> X;
  constexpr int kLanes = F::kGroup / 8;  // of a group
  const int qbits = digits == 4 ? 26 : 19;  // |q| <= 2^qbits keeps the top digit within a signed byte
  float s[R], mx[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    s[r] = ((v[r][0] + v[r][1]) + (v[r][2] + v[r][3])) + ((v[r][4] + v[r][5]) + (v[r][6] + v[r][7]));
    mx[r] = max_nan(max_nan(max_nan(fabsf(v[r][0]), fabsf(v[r][1])), max_nan(fabsf(v[r][2]), fabsf(v[r][3]))),
                    max_nan(max_nan(fabsf(v[r][4]), fabsf(v[r][5])), max_nan(fabsf(v[r][6]), fabsf(v[r][7]))));
  }
#pragma unroll
  for (int o = SPLIT; o < kLanes * SPLIT; o <<= 1) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (F::kSums) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
      mx[r] = max_nan(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], o));
    }
  }
  const int sub = lane % SPLIT;
  lane /= SPLIT;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    int e = (int)((__float_as_uint(mx[r]) >> 23) & 0xFF);  // mx < 2^(e-126)
    const bool finite = e < 255, tiny = e < qbits;  // (whose elements want a factor above 2^127)
    if (e < qbits - 23) e = qbits - 23;             // units of 2^-149, as fine as floats get
    if (e > 254) e = 254;
    if (sub == 0 && lane % kLanes == 0) {
      float* tab = reinterpret_cast<float*>(xb[r] + X::kFrag);
      const int g = lane / kLanes;
      const int f = e - 126 - qbits + 127;  // 2^(E-qbits)
      const float sc[2] = {finite ? pow2_biased(f) : __uint_as_float(0x7FC00000u), finite ? pow2_biased(f + 14) : __uint_as_float(0x7FC00000u)};
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float* t = tab + X::entry(m[r], p, g);
        t[0] = sc[p];
        if (F::kSums) t[1] = p ? s[r] : 0.f;
      }
    }
    const float fi = __uint_as_float((uint32_t)(qbits - (e - 126) + 127 - (tiny ? 64 : 0)) << 23);
    const uint32_t bias = digits == 4 ? 64u * (1 + 128 + 16384) : 64u * (1 + 128);
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) y[i] = v[r][i];
    if (tiny) {
#pragma unroll
      for (int i = 0; i < 8; ++i) y[i] *= 18446744073709551616.f;  // 2^64: exact
    }
    int q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = (int)((uint32_t)__float2int_rn(y[i] * fi) + bias);
    auto digit = [&](int d) {
      uint32_t p[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        auto at = [&](int i) { return (uint32_t)(q[F::kWords ? 2 * i + h : 4 * h + i] >> (7 * d)); };
        p[h] = __byte_perm(__byte_perm(at(0), at(1), 0x0040), __byte_perm(at(2), at(3), 0x0040), 0x5410);
        if (d < digits - 1) {
          p[h] = (p[h] & 0x7F7F7F7Fu) ^ 0x40404040u;
          p[h] |= (p[h] & 0x40404040u) << 1;
        }
        if (d >= digits) p[h] = 0;
      }
      return make_uint2(p[0], p[1]);
    };
    const int step = lane >> 2, w = lane & 3;  // the lane's eight positions are 8 w .. 8 w + 7 of the K step
    auto put_at = [&](int n, uint2 t) {
      if (F::kWords) {  // the nibbles' order: even elements of a packed word, then odd ones
        *reinterpret_cast<uint2*>(xb[r] + X::frag(step, n, w)) = t;
      } else {
        *reinterpret_cast<uint32_t*>(xb[r] + X::frag(step, n, 2 * (w & 1)) + 4 * (w >> 1)) = t.x;
        *reinterpret_cast<uint32_t*>(xb[r] + X::frag(step, n, 2 * (w & 1) + 1) + 4 * (w >> 1)) = t.y;
      }
    };
    const int half = FMT == FMT_MLX4 ? (step >> 1) & 1 : FMT == FMT_Q6K ? w >> 1 : step & 1;
    auto put = [&](int d, uint2 t) {
      if (MB > 1) {
        put_at(m[r] * 4 + d, t);
      } else {
        put_at(half * 4 + d, t);
        put_at((half ^ 1) * 4 + d, make_uint2(0, 0));
      }
    };
    if (SPLIT == 4) {
      put(sub, digit(sub));
    } else {
#pragma unroll
      for (int d = 0; d < 4; ++d) put(d, digit(d));
    }
  }
}
// FP8: the chunk is scaled by a power of two so that its largest magnitude lies in [128, 256) and every element written as six e4m3
// values, each the rounding of what those before it left (exact in f32), the remainder times 2^8 after every second one: an f32
// exactly, down to 2^-32 of the chunk's largest element.  Column p of the row's tile holds piece p; the table has, per lane of a quad, the scale of
// its two columns.  (Chunks below 2^-120 are scaled as if they had an element of that size, which leaves their elements exact down to the
// smallest subnormal; the scales of their last pieces, down to 2^-143, are subnormal themselves.)
template <int MB>
__device__ __forceinline__ void prep_fp8(const float (&v)[8], int lane, unsigned char* xb, int m) {
  typedef XBlock<FMT_FP8, MB> X;
  float mx = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) mx = max_nan(mx, fabsf(v[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max_nan(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  int e = (int)((__float_as_uint(mx) >> 23) & 0xFF) - 127;
  const bool finite = e < 128;
  if (e < -120) e = -120;
  if (e > 127) e = 127;
  const float s = __uint_as_float((uint32_t)(7 - e + 127) << 23);
  if (lane < 3) reinterpret_cast<float*>(xb + X::kFrag)[m * 4 + lane] = finite ? pow2_biased(e - 7 - 8 * lane + 127) : __uint_as_float(0x7FC00000u);
  float r[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = v[i] * s;
  const int step = lane >> 2, w = lane & 3;
#pragma unroll
  for (int p = 0; p < 6; ++p) {
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      unsigned short b;
      asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b) : "f"(r[2 * i + 1]), "f"(r[2 * i]));
      uint32_t f;
      asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(f) : "h"(b));
      r[2 * i] -= f16_lo(f);
      r[2 * i + 1] -= f16_hi(f);
      h[i] = b;
    }
    if (p & 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i) r[i] *= 256.f;
    }
    const int n = m * 8 + p;
    *reinterpret_cast<uint32_t*>(xb + X::frag(step, n, 2 * (w & 1)) + 4 * (w >> 1)) = h[0] | (h[1] << 16);
    *reinterpret_cast<uint32_t*>(xb + X::frag(step, n, 2 * (w & 1) + 1) + 4 * (w >> 1)) = h[2] | (h[3] << 16);
  }
}
template <int FMT, int MB, int SPLIT = 1>
__device__ __forceinline__ void prep_chunk(const float (&v)[8], int lane, unsigned char* xb, int m, int digits) {
  if constexpr (FMT == FMT_FP8) {
    prep_fp8<MB>(v, lane, xb, m);
    return;
  }
  unsigned char* const xbs[1] = {xb};
  const int ms[1] = {m};
  prep_chunks<FMT, MB, SPLIT, 1>(reinterpret_cast<const float(&)[1][8]>(v), lane, xbs, ms, digits);
}
__device__ __forceinline__ void load_eight(const float* p, float (&v)[8]) {
  if ((reinterpret_cast<uintptr_t>(p) & 15) == 0) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {  // callers may hand in x at any float
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = p[i];
  }
}

// The launch in front of the product: a block per (activation row, chunk).
template <int FMT, int MB>
__global__ void __launch_bounds__(128)
mlx_prep_x_kernel(const float* __restrict__ x, unsigned char* __restrict__ xb, int in_dim, int digits) {
  const int nchunks = (in_dim + kChunkK - 1) / kChunkK, m = blockIdx.x / nchunks, c = blockIdx.x - m * nchunks, lane = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();  // x may be the output of the kernel in front
  float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // (past the row)
  if constexpr (FMT == FMT_FP8) {  // (a block of one warp)
    const int k = c * kChunkK + lane * 8;
    if (k < in_dim) load_eight(x + (size_t)m * in_dim + k, v);
    prep_fp8<MB>(v, lane, xb + (size_t)c * XBlock<FMT, MB>::kBytes, m);
    return;
  }
  const int k = c * kChunkK + lane / 4 * 8;
  if (k < in_dim) load_eight(x + (size_t)m * in_dim + k, v);
  prep_chunk<FMT, MB, 4>(v, lane, xb + (size_t)c * XBlock<FMT, MB>::kBytes, m, digits);
}

// ---- the product kernel ----------------------------------------------------------------------------

__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// D = A * B + C, 16 x 8 x 32 (bytes), s32.
template <bool SIGNED>
__device__ __forceinline__ void imma32(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int c0, int c1, int c2, int c3) {
  if (SIGNED)
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
  else
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
// D = A * B + C, 16 x 8 x 16.
__device__ __forceinline__ void imma16(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0, int c) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(b0), "r"(c));
}
// D = A * B + D, 16 x 8 x 32, e4m3, f32 (an MMA's error is that of f32: 3e-7 of its largest term at most, measured).
__device__ __forceinline__ void qmma32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.f32.e4m3.e4m3.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The accumulators start at 1.5 * 2^23 as a float's bits, so that an integer sum v below 2^22 in magnitude comes out as the
// float 1.5 * 2^23 + v, without a conversion; two digits' sums then meet exactly (both terms are multiples of 128 or below 2^24).
constexpr int kAcc0 = 0x4B400000;
constexpr float kAcc0F = 12582912.f;
__device__ __forceinline__ float digits_sum(int lo, int hi) { return fmaf(__int_as_float(hi), 128.f, -129.f * kAcc0F) + __int_as_float(lo); }


// The scales of a chunk's rows.  K-quants pack them in six bits or multiply them by the super-block's d.  fma(2^23 + field, d,
// -2^23 d) is the product field * d rounded once, as the reference's dequantisation does.  With one row of x a lane finishes half
// of its rows' blocks and unpacks those itself; with several a warp's lanes unpack every block once (two lanes a row) and leave
// {scale, minimum} in shared memory, a row 80 bytes apart, so that eight rows lie in different banks.  (One row, that way: Q4_K
// 128256x4096 61 us a call, 51 by every lane for itself; two rows, 14336x4096 11.8 and 13.3.)
template <int FMT, int MB>
constexpr bool kStaged = MB > 1 && (FMT == FMT_Q4K || FMT == FMT_Q5K || FMT == FMT_Q6K);
constexpr int kStagedRow = 80;

template <int FMT>
__device__ __forceinline__ void stage_scales(const unsigned char* st, int row, unsigned char* dst, int lane) {  // 16 rows from `row`
  const int r = lane >> 1, q = lane & 1;  // this lane: the row's blocks of the chunk's half q
  const unsigned char* p = st + Fmt<FMT>::kStageWBytes + (row + r) * Fmt<FMT>::kMetaRow;
  unsigned char* d = dst + r * kStagedRow + 32 * q;
  float v[8];
  if (FMT == FMT_Q6K) {  // bytes 8 q .. 8 q + 7
    const uint2 w = *reinterpret_cast<const uint2*>(p + 8 * q);
    const float dd = 0.25f * __half2float(*reinterpret_cast<const __half*>(st + Fmt<FMT>::kDOff + (row + r) * 2));  // (the bytes are 4 (q - 32))
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(dd, __uint_as_float(__byte_perm((k < 4 ? w.x : w.y) ^ 0x80808080u, 0x4B000000u, 0x7440u + (k & 3))) - 8388736.f);
  } else {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const float dd = f16_lo(w.x), dm = f16_hi(w.x) * -0.015625f, kd = dd * -8388608.f, km = dm * -8388608.f;
    const uint32_t lo = q ? __funnelshift_r(w.z, w.w, 16) : w.y, hi = q ? w.w >> 16 : w.z;  // 48 bits
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t f = k == 0 ? lo : k == 1 ? lo >> 12 : k == 2 ? __funnelshift_r(lo, hi, 24) : hi >> 4;
      v[2 * k] = fmaf(__uint_as_float((f & 63u) | 0x4B000000u), dd, kd);
      v[2 * k + 1] = fmaf(__uint_as_float((f & 0xFC0u) | 0x4B000000u), dm, km);  // (2^23 + 64 m) * (-dmin / 64) + ...
    }
  }
  *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(d + 16) = make_float4(v[4], v[5], v[6], v[7]);
}

// One row of x: what a lane keeps of a row's scale data, and scale and minimum of its block of pair j (bit 24 j + 12 half of the
// packed fields; Q6_K: byte 2 j + half).
template <int FMT>
struct RowScales {
  uint4 w;
  float d, kd, m, km;
  __device__ __forceinline__ void load(const unsigned char* st, int row) {
    w = *reinterpret_cast<const uint4*>(st + Fmt<FMT>::kStageWBytes + row * Fmt<FMT>::kMetaRow);
    if (FMT == FMT_Q6K) {
      d = 0.25f * __half2float(*reinterpret_cast<const __half*>(st + Fmt<FMT>::kDOff + row * 2));
      w.x ^= 0x80808080u;
      w.y ^= 0x80808080u;
      w.z ^= 0x80808080u;
      w.w ^= 0x80808080u;
    } else if (FMT != FMT_Q80) {
      d = f16_lo(w.x);
      m = f16_hi(w.x) * -0.015625f;
      kd = d * -8388608.f;
      km = m * -8388608.f;
    }
  }
  __device__ __forceinline__ float2 pair(int j, int half) const {
    if (FMT == FMT_Q80) return make_float2(f16_lo((j == 0 ? w.x : j == 1 ? w.y : j == 2 ? w.z : w.w) >> (16 * half)), 0.f);
    if (FMT == FMT_Q6K) {
      const uint32_t b = __byte_perm((j >> 1) == 0 ? w.x : (j >> 1) == 1 ? w.y : (j >> 1) == 2 ? w.z : w.w, 0x4B000000u, 0x7440u + 2 * (j & 1) + half);
      return make_float2(__fmul_rn(d, __uint_as_float(b) - 8388736.f), 0.f);
    }
    const int sh = 12 * half;
    const uint32_t f = j == 0 ? w.y >> sh : j == 1 ? __funnelshift_r(w.y, w.z, 24) >> sh : j == 2 ? __funnelshift_r(w.z, w.w, 16) >> sh : w.w >> (sh + 8);
    return make_float2(fmaf(__uint_as_float((f & 63u) | 0x4B000000u), d, kd), fmaf(__uint_as_float((f & 0xFC0u) | 0x4B000000u), m, km));
  }
};

// One weight of a launch.
struct RowSeg {
  const unsigned char* w;  // weight blocks [tile][chunk]; row-major FP8: the bytes (row-major MLX: by its tensor maps only)
  float* out;              // [batch][out_dim]
  int out_dim, tile0;      // first of its tiles among the launch's
  const float *scale, *bias;  // FP8: [out_dim]; [out_dim] or nullptr
};
constexpr int kMaxRowSeg = 4;

struct MmaArgs {
  RowSeg seg[kMaxRowSeg];
  int nseg;
  const float* x;          // [batch][in_dim]
  const unsigned char* xb; // prepared activations: an XBlock per chunk
  int* status;             // device word: 0 ok, otherwise the first wait that gave up
  float* scratch;          // split-K partial sums [item][warp][value][lane]
  unsigned int* counters;  // arrival counters per tile and warp, zero between launches
  int in_dim;
  int batch;               // activation rows of this launch (<= MB of the instantiation)
  int digits;
  int ntiles;              // tiles of 128 rows, of all weights
  int nchunks;             // ceil(in_dim / 256)
  int splits;              // CTAs sharing the K range of one tile
  int items;               // ntiles * splits
  int stages;              // depth of the shared-memory ring
  int cmax;                // FUSED: most chunks an item has (resident XBlocks)
  int cluster;             // the CTAs of a tile are a cluster and have one item each
  int plain;               // outputs of an activation row with a NaN or an infinity are those of f32 products (see plain_product); else all NaN
  const MmaGroupEntry* gwork;
  const int* gcount;
  int gmax, gtpe, gmats, gfirst, gdirect;
  size_t gxb;
};

// Where element k of a stage's row r lies in the nibble image of Q5_K and Q6_K: byte, and whether in the high nibble; the bits beside it.
__device__ __forceinline__ int kq_byte(int r, int k) { return r * 128 + (((k >> 5) ^ (r & 7)) << 4) + (k & 15); }
__device__ __forceinline__ bool kq_upper(int k) { return (k & 16) != 0; }
__device__ __forceinline__ int q5k_bit_byte(int r, int k) { return Fmt<FMT_Q5K>::kHighOff + (k >> 7) * 2048 + r * 16 + (k & 15); }
__device__ __forceinline__ int q5k_bit(int k) { return 2 * ((k >> 5) & 3) + ((k >> 4) & 1); }
__device__ __forceinline__ int q6k_bits_byte(int r, int k) { return Fmt<FMT_Q6K>::kHighOff + (k >> 6) * 2048 + r * 16 + (k & 15); }
__device__ __forceinline__ int q6k_bits(int k) { return 4 * ((k >> 5) & 1) + 2 * ((k >> 4) & 1); }

// Weight k of a stage's row r, rounded as the reference's dequantisation does (loader/gguf/quant_matrix.go:138-158, :378-426).
template <int FMT>
__device__ __forceinline__ float tiled_weight(const unsigned char* stg, int r, int k) {
  if (FMT == FMT_Q80) {
    const signed char q = (signed char)stg[(k >> 5) * 4096 + ((k >> 4) & 1) * 2048 + (r >> 3) * 128 + (r & 7) * 16 + (k & 15)];
    return __fmul_rn(__half2float(*reinterpret_cast<const __half*>(stg + Fmt<FMT_Q80>::kStageWBytes + r * 16 + (k >> 5) * 2)), (float)q);
  }
  const float d = __half2float(*reinterpret_cast<const __half*>(stg + Fmt<FMT_Q6K>::kDOff + r * 2));
  const signed char sc = (signed char)stg[Fmt<FMT_Q6K>::kStageWBytes + r * 16 + (k >> 4)];
  const uint32_t low = (stg[kq_byte(r, k)] >> (kq_upper(k) ? 4 : 0)) & 0xFu, two = (stg[q6k_bits_byte(r, k)] >> q6k_bits(k)) & 3u;
  return __fmul_rn(__fmul_rn(d, (float)sc), (float)((int)(low | (two << 4)) - 32));
}

// A row with an infinity: its digits are NaN, and so is what the tensor cores give.  Formats without minima have an answer all the same, an infinity of the weight's
// sign (NaN where two meet or the weight is zero), and the kernels for other numbers of rows give it.  Launches that share a weight with those look at their NaN
// outputs again: if the activation row is not finite, the lane takes the f32 products of its weight row one after another.  (A NaN code of an FP8 weight costs the scan
// of the activations only.)
__device__ __forceinline__ bool row_is_finite(const float* x, int n, int lane) {  // by a warp
  bool ok = true;
  for (int k = lane; k < n; k += 32) ok = ok && (__float_as_uint(x[k]) & 0x7F800000u) != 0x7F800000u;
  return __all_sync(0xffffffffu, ok);
}
template <int FMT, bool TILED>
__device__ float plain_product(const unsigned char* w, const float* x, int row, int in_dim, int nchunks) {
  float acc = 0.f;
  if (FMT == FMT_FP8) {
    for (int k = 0; k < in_dim; ++k) {
      uint32_t f;
      asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(f) : "h"((unsigned short)w[(size_t)row * in_dim + k]));
      acc = fmaf(f16_lo(f), x[k], acc);
    }
    return acc;
  }
  const int r = row & (kTileRows - 1);
  for (int c = 0; c < nchunks; ++c) {
    const unsigned char* st = w + ((size_t)(row / kTileRows) * nchunks + c) * Fmt<FMT>::kStageBytes;
    for (int k = 0; k < kChunkK && c * kChunkK + k < in_dim; ++k) acc = fmaf(tiled_weight<FMT>(st, r, k), x[c * kChunkK + k], acc);
  }
  return acc;
}

// Row-major weights: their tiles come as boxes of 128 rows, 128 bytes of nibbles (whose 128-byte swizzle is the tiled image's) and
// 16 bytes of the table, or twice 128 bytes (FP8); zeros past the edges.
struct RowMaps {
  CUtensorMap map[kMaxRowSeg][2];
};
struct NoMaps {};
template <bool TILED>
using MapArgs = std::conditional_t<TILED, NoMaps, RowMaps>;
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
template <bool G, bool WORK = false>
struct StageWalkT {
  int w, tile, split, c, c1;
  int wend, entry, mat;  // G only
  __device__ __forceinline__ void open(const MmaArgs& a) {
    if (G) {
      const int per = a.gtpe * a.gmats;
      entry = w / per;
      const int rem = w - entry * per;
      mat = rem / a.gtpe;
      tile = rem - mat * a.gtpe;
      if (WORK && a.gdirect == 2) {  // gate and up of a tile one behind the other
        mat = rem & 1;
        tile = rem >> 1;
      }
      split = 0;
      c = 0;
      c1 = a.nchunks;
    } else {
      tile = w / a.splits;
      split = w - tile * a.splits;
      c = split * a.nchunks / a.splits;
      c1 = (split + 1) * a.nchunks / a.splits;
    }
  }
  __device__ __forceinline__ StageWalkT(const MmaArgs& a, int live_items = 0) : w(blockIdx.x) {
    if (G) {
      const int each = WORK && a.gdirect == 2 ? 2 : 1;  // (whole pairs)
      w = (int)((long long)blockIdx.x * (live_items / each) / gridDim.x) * each;
      wend = (int)((long long)(blockIdx.x + 1) * (live_items / each) / gridDim.x) * each;
    }
    if (live(a)) open(a);
  }
  __device__ __forceinline__ bool live(const MmaArgs& a) const { return G ? w < wend : w < a.items; }
  __device__ __forceinline__ void next_item(const MmaArgs& a) {
    w += G ? 1 : gridDim.x;
    if (live(a)) open(a);
  }
};

constexpr int kConsumers = 8;  // warps; the ninth loads
constexpr int kMaxStages = 12, kMaxSplits = 16;
constexpr int kThreads = (kConsumers + 1) * 32;

template <int FMT, int MB, bool G>
struct RowCfg {
  // Sixteen rows a warp, or 32 with the warps in two groups that take turns at the stages: fragments of several n tiles are
  // read from shared memory half as often.
  static constexpr int SL = (FMT != FMT_FP8 && MB >= 4) || G ? 2 : 1, KG = SL;  // (FP8: a tile of sums for every activation row is registers enough)
  static constexpr int NT = XBlock<FMT, MB>::NT;
  static constexpr int kVals = SL * NT;                      // values a lane has of an item
  static constexpr int kStoring = kConsumers / KG;           // warps that finish items
  static constexpr int kPair = KG == 2 ? 2 * kStoring * kVals * 128 : 0;
  static constexpr int kRecv = kStoring * kVals * 128;       // a split's sums
  static constexpr int kScales = kStaged<FMT, MB> ? kConsumers * SL * 16 * kStagedRow : 0;
};
// A warp's outputs of a tile, of which some are NaN (see plain_product); row: of the lane's first output.  Called once, where the kernel ends.
template <int FMT, int MB, bool TILED, int VALS>
__device__ __forceinline__ void store_again(const MmaArgs& a, int sg, int row, int lane) {
  typedef XBlock<FMT, MB> X;
  constexpr int kHalves = MB > 1 && !X::kRowTile ? 2 : 1;  // activation rows that a warp has values of at a time
  const int t = lane & 3;
  const RowSeg& w = a.seg[sg];
  for (int k = 0; k < VALS; ++k) {
    const int r = row + 16 * (k / X::NT), m0 = MB == 1 ? 0 : kHalves * (k % X::NT), m = m0 + (kHalves == 2 ? t >> 1 : 0);
    float* const out = w.out + (size_t)m * w.out_dim + r;
    const bool odd = (t < 2 || kHalves == 2) && m < a.batch && r < w.out_dim && isnan(*out);
    if (!__any_sync(0xffffffffu, odd)) continue;
    bool finite = true;
    for (int h = 0; h < kHalves; ++h) {
      if (m0 + h >= a.batch) continue;
      const bool f = row_is_finite(a.x + (size_t)(m0 + h) * a.in_dim, a.in_dim, lane);
      if (m0 + h == m) finite = f;
    }
    if (odd && !finite) {
      const float v = plain_product<FMT, TILED>(w.w, a.x + (size_t)m * a.in_dim, r, a.in_dim, a.nchunks);
      *out = FMT == FMT_FP8 ? fmaf(v, w.scale[r], w.bias ? w.bias[r] : 0.f) : v;
    }
    __syncwarp();
  }
}

template <int FMT, int MB, bool FUSED, bool G, bool TILED = true>
struct RowSmem {
  static constexpr int kStage = Fmt<FMT>::kStageBytes + (FUSED ? 0 : XBlock<FMT, MB>::kBytes);
  static __host__ __device__ size_t bytes(int stages, int cmax, int recv) {
    return (size_t)stages * kStage + (FUSED ? (size_t)cmax * XBlock<FMT, MB>::kBytes : 0) + RowCfg<FMT, MB, G>::kPair + RowCfg<FMT, MB, G>::kScales + (size_t)recv * RowCfg<FMT, MB, G>::kRecv + 512 +
           (TILED ? 0 : 1024);  // (boxes with a swizzle start on multiples of 1024 bytes)
  }
  // Depth of the ring that `budget` leaves room for.
  static int stages(size_t budget, int cmax, int recv) {
    const size_t fixed = bytes(0, cmax, recv);
    int n = fixed < budget ? (int)((budget - fixed) / kStage) : 0;
    if (n > kMaxStages) n = kMaxStages;
    return RowCfg<FMT, MB, G>::KG == 2 ? n & ~1 : n;  // (a group must see every round of its slots)
  }
};

// Formats without minima, three rows and more: launches have an SM to a CTA always (launch_one), which leaves registers for two sums of every value.
template <int FMT, int MB, bool G>
constexpr bool kAlone = (FMT == FMT_Q80 || FMT == FMT_Q6K) && MB >= 4 && !G;

template <int FMT, int MB, bool FUSED, bool G = false, bool TILED = true>
__global__ void __launch_bounds__(kThreads, kAlone<FMT, MB, G> ? 1 : 2)
mlx_mma_kernel(const __grid_constant__ MmaArgs a, const __grid_constant__ MapArgs<TILED> maps) {
  static_assert(!G || !FUSED, "grouped launches: activations prepared in front");
  static_assert(TILED || ((FMT == FMT_MLX4 || FMT == FMT_FP8) && FUSED), "row-major: MLX and FP8, activations by the CTAs themselves");
  constexpr bool kWork = G && FMT != FMT_MLX4;  // a work list's entries (MmaWorkEntry)
  typedef StageWalkT<G, kWork> StageWalk;
  typedef Fmt<FMT> F;
  typedef XBlock<FMT, MB> X;
  typedef RowCfg<FMT, MB, G> C;
  typedef RowSmem<FMT, MB, FUSED, G, TILED> M;
  constexpr int SL = C::SL, KG = C::KG, NT = C::NT, kStage = M::kStage;
  // A chunk is summed by itself: its terms, products and biases or minima that cancel, meet a small sum, and without minima the lane's sum has a sixteenth or an
  // eighth of the terms (errors against 64 bits, as one sum / so: Q6_K 28672x8192 two rows 4.0e-7 / 1.3e-7, 4096x4096 1.5e-7 / 1.0e-7, Q8_0 2.9e-7 / 1.1e-7; the kernels
  // that these came from: 2.9e-7, 1.2e-7 and 2.1e-7).
  constexpr bool kByChunk = FMT != FMT_FP8 && !(FMT == FMT_MLX4 && MB == 8) && !(FMT == FMT_Q80 && G);
  extern __shared__ __align__(128) unsigned char smem_dyn[];
  const int S = a.stages;
  unsigned char* ring = TILED ? smem_dyn : reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  unsigned char* bres = ring + (size_t)S * kStage;
  unsigned char* scales = bres + (FUSED ? (size_t)a.cmax * X::kBytes : 0);
  float* pair = reinterpret_cast<float*>(scales + C::kScales);
  float* recv = pair + C::kPair / 4;
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<unsigned char*>(recv) + (a.cluster ? (size_t)(a.splits - 1) * C::kRecv : 0));
  volatile int* gave_up = reinterpret_cast<volatile int*>(bars + 2 * S);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * S;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, kConsumers / KG);
    }
    for (int s = 0; s < 9; ++s) gave_up[s] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (!G) pdl_launch_dependents();
  __syncthreads();
  if (a.cluster) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (waited for before the first store to a peer: it has started)
  bool ok = true;
  int gitems = 0;
  if (G) {
    pdl_wait();  // the work entries come from the kernels in front
    int n = __ldcg(a.gcount);
    if (n > a.gmax) n = a.gmax;
    gitems = n * a.gtpe * a.gmats;
  }
  StageWalk sw(a, gitems);
  auto entry_at = [&](int e) -> const MmaGroupEntry* {
    return kWork ? &reinterpret_cast<const MmaWorkEntry*>(a.gwork)[e].g : a.gwork + e;
  };
  const int cbase = sw.live(a) ? sw.c : 0;  // first chunk of this CTA's K range
  auto finish = [&](int k, int r, float v) {
    if (FMT != FMT_FP8) return v;
    const float* bias = a.seg[k].bias;
    return fmaf(v, __ldg(a.seg[k].scale + r), bias ? __ldg(bias + r) : 0.f);
  };
  auto seg_of = [&](int tile) {
    int k = 0;
#pragma unroll
    for (int j = 1; j < kMaxRowSeg; ++j)
      if (j < a.nseg && tile >= a.seg[j].tile0) k = j;
    return k;
  };
  float fin[C::kVals];                      // the item's values (cluster: kept for the exchange)
  bool have = false;
  constexpr bool kPlain = !G && (TILED ? FMT == FMT_Q80 || FMT == FMT_Q6K : FMT == FMT_FP8);
  uint32_t odd = 0;  // items of which this lane has stored a NaN (bit 31: or a later one; where K is cut and sums meet in scratch a CTA has at most 10)

  if (warp == kConsumers) {
    // ------------------------------------------------------------------ producer
    if constexpr (!TILED) {
      if (lane == 0) {
        RingCursor rc;
        int i = 0;
        for (; sw.live(a) && ok; sw.next_item(a)) {
          const int k = seg_of(sw.tile), row0 = (sw.tile - a.seg[k].tile0) * kTileRows;
          for (int c = sw.c; c < sw.c1; ++c, ++i, rc.next(S)) {
            if (i >= S) ok = mbar_wait(empty0 + 8 * rc.s, rc.ph ^ 1u, a.status, 1);
            if (!ok) break;
            const uint32_t dst = smem_u32(ring + (size_t)rc.s * kStage), bar = full0 + 8 * rc.s;
            mbar_expect_tx(bar, F::kStageBytes);
            if (FMT == FMT_FP8) {
              tma_load_2d(dst, &maps.map[k][0], c * 256, row0, bar);
              tma_load_2d(dst + 16384, &maps.map[k][0], c * 256 + 128, row0, bar);
            } else {
              tma_load_2d(dst, &maps.map[k][0], c * 128, row0, bar);
              tma_load_2d(dst + F::kStageWBytes, &maps.map[k][1], c * 16, row0, bar);
            }
          }
        }
        if (!ok) *gave_up = 1;
      }
    } else if (lane == 0) {
      auto wsrc = [&](const StageWalk& s, int c) {
        const unsigned char* base;
        int tile = s.tile;
        if (!G) {
          const int k = seg_of(tile);
          base = a.seg[k].w;
          tile -= a.seg[k].tile0;
        }
        if (G) base = reinterpret_cast<const unsigned char*>(__ldg(reinterpret_cast<const unsigned long long*>(&entry_at(s.entry)->w[a.gfirst + s.mat])));
        return base + ((size_t)tile * a.nchunks + c) * F::kStageBytes;
      };
      auto bsrc = [&](const StageWalk& s, int c) { return a.xb + (G ? (size_t)s.entry * a.gxb : 0) + (size_t)c * X::kBytes; };
      // The weights do not depend on the kernel in front: the ring is filled with them first, the activations of those
      // stages follow when they are there.
      RingCursor rc;
      int i = 0;
      bool waited = FUSED || G;
      StageWalk sx = sw;  // the first stage whose activations have not been asked for
      int xc = sx.c, xi = 0;
      auto catch_up = [&] {
        pdl_wait();
        waited = true;
        for (; xi < i; ++xi) {
          bulk_load_1d(smem_u32(ring + (size_t)xi * kStage) + F::kStageBytes, bsrc(sx, xc), X::kBytes, full0 + 8 * xi);
          if (++xc == sx.c1) {
            sx.next_item(a);
            xc = sx.c;
          }
        }
      };
      for (; sw.live(a) && ok; sw.next_item(a)) {
        for (int c = sw.c; c < sw.c1; ++c, ++i, rc.next(S)) {
          if (i == S && !waited) catch_up();
          if (i >= S) ok = mbar_wait(empty0 + 8 * rc.s, rc.ph ^ 1u, a.status, 1);
          if (!ok) break;
          const uint32_t dst = smem_u32(ring + (size_t)rc.s * kStage), bar = full0 + 8 * rc.s;
          mbar_expect_tx(bar, kStage);
          bulk_load_1d(dst, wsrc(sw, c), F::kStageBytes, bar);
          if (!FUSED && waited) bulk_load_1d(dst + F::kStageBytes, bsrc(sw, c), X::kBytes, bar);
        }
      }
      if (!waited) catch_up();
      if (!ok) *gave_up = 1;
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ consumers
    const int g = lane >> 2, t = lane & 3, half = t >> 1, p = t & 1;
    const int grp = KG == 2 ? warp >> 2 : 0, slot = KG == 2 ? warp & 3 : warp;  // slot: of the warps that finish items
    const int row0 = slot * (16 * SL);
    if (FUSED) {
      pdl_wait();
      // every item of this CTA covers the same K range (the grid is a multiple of the K splits)
      if (sw.live(a)) {
        const int n = sw.c1 - sw.c;
        auto load = [&](int i, float (&v)[8]) {
          const int m = MB == 1 ? 0 : i / n, k = (sw.c + i - m * n) * kChunkK + lane * 8;
          if (k < a.in_dim) {
            load_eight(a.x + (size_t)m * a.in_dim + k, v);
          } else {  // (past the row, which ends with a lane's eight)
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.f;
          }
        };
        float v[8];
        if (warp < a.batch * n) load(warp, v);
#pragma unroll 1
        for (int i = warp; i < a.batch * n; i += kConsumers) {
          float u[8] = {};
          if (i + kConsumers < a.batch * n) load(i + kConsumers, u);  // (the next chunk is under way while this one is worked on)
          const int m = MB == 1 ? 0 : i / n;
          prep_chunk<FMT, MB>(v, lane, bres + (size_t)(i - m * n) * X::kBytes, m, a.digits);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = u[e];
        }
      }
      asm volatile("bar.sync 1, %0;" ::"n"(kConsumers * 32) : "memory");
    }
    // shared-memory addresses that stay: of the lane's rows in an ldmatrix (nibbles: two K steps of 16 rows; bytes: one), and
    // of its part of the fragments and tables
    const int mi = lane >> 3, lr = lane & 7;
    const uint32_t a_lane = F::kNibble || !TILED ? (row0 + (mi & 1) * 8 + lr) * 128 : (mi >> 1) * 2048 + (row0 / 8 + (mi & 1)) * 128 + lr * 16;
    const uint32_t b_lane = lane * 16;
    const int t_lane = X::kFrag + 4 * (FMT == FMT_FP8 ? t : MB > 1 ? X::entry(half, p, 0) : X::entry(0, p, FMT == FMT_Q6K ? 0 : half));
    const bool mine = t < 2 || (MB > 1 && !X::kRowTile);
    auto act = [&](int k) { return MB == 1 ? 0 : X::kRowTile ? k % NT : 2 * (k % NT) + half; };
    auto store = [&](int tile, int item, auto&& value) {  // the warp's values of a tile, by the warp as one
      const int sg = seg_of(tile), row = (tile - a.seg[sg].tile0) * kTileRows + row0 + g + 8 * p, out_dim = a.seg[sg].out_dim;
      float* const out = a.seg[sg].out;
      bool nan = false;
#pragma unroll
      for (int k = 0; k < C::kVals; ++k) {
        const int m = act(k), r = row + 16 * (k / NT);
        const float v = value(k);
        if (mine && m < a.batch && r < out_dim) {  // (of rows past the batch the digits are whatever was there)
          nan = nan || isnan(v);
          out[(size_t)m * out_dim + r] = finish(sg, r, v);
        }
      }
      if (kPlain && nan) odd |= 1u << (item < 31 ? item : 31);
    };
    unsigned char* sc_warp = scales + warp * (SL * 16 * kStagedRow);
    float gate[kWork ? C::kVals : 1];
    int cur_entry = -1, nb = a.batch;
    RingCursor rc;
    int i = 0, items = 0;
    for (; sw.live(a) && ok; sw.next_item(a), ++items) {
      float acc[SL][NT][2], before[kByChunk ? SL : 1][kByChunk ? NT : 1][2];
#pragma unroll
      for (int sl = 0; sl < SL; ++sl)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[sl][nt][0] = acc[sl][nt][1] = 0.f;
      float low[FMT == FMT_FP8 ? SL : 1][FMT == FMT_FP8 ? NT : 1][2] = {};
#pragma unroll 1
      for (int c = sw.c; c < sw.c1; ++c, ++i, rc.next(S)) {
        if (KG == 2 && (i & 1) != grp) continue;
        ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * rc.s, rc.ph, a.status, 4));
        if (!ok) break;
        if constexpr (kByChunk) {
#pragma unroll
          for (int sl = 0; sl < SL; ++sl)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                before[sl][nt][r] = acc[sl][nt][r];
                acc[sl][nt][r] = 0.f;
              }
        }
        const unsigned char* st = ring + (size_t)rc.s * kStage;
        const unsigned char* xb = FUSED ? bres + (size_t)(c - cbase) * X::kBytes : st + F::kStageBytes;
        const uint32_t st_a = smem_u32(st) + a_lane;
        const unsigned char* xf = xb + b_lane;
        const unsigned char* xt = xb + t_lane;
        if constexpr (kStaged<FMT, MB>) {
#pragma unroll
          for (int sl = 0; sl < SL; ++sl) stage_scales<FMT>(st, row0 + 16 * sl, sc_warp + sl * (16 * kStagedRow), lane);
          __syncwarp();
        }
        const unsigned char* sc_lane = sc_warp + g * kStagedRow;
        const unsigned char* meta = st + F::kStageWBytes + (row0 + g) * F::kMetaRow;
        RowScales<FMT> rs[MB == 1 ? SL : 1][2];
        if constexpr (MB == 1 && FMT != FMT_MLX4) {
#pragma unroll
          for (int sl = 0; sl < SL; ++sl)
#pragma unroll
            for (int r = 0; r < 2; ++r) rs[sl][r].load(st, row0 + 16 * sl + 8 * r + g);
        }
        // scales (and biases) of the rows g + 8 r of slab sl
        auto mlx_scale = [&](int sl, int r, int word, float& sv, float& bv) {  // word: per lane
          const uint32_t w = *reinterpret_cast<const uint32_t*>(meta + (16 * sl + 8 * r) * 16 + 4 * word);
          sv = __uint_as_float(w << 16);
          bv = __uint_as_float(w & 0xFFFF0000u);
        };
        // A fragments of K step s
        uint32_t af[SL][2][4], high[FMT == FMT_Q5K || FMT == FMT_Q6K ? SL : 1][4];
        auto load_a = [&](int j) {  // both steps of pair j
#pragma unroll
          for (int sl = 0; sl < SL; ++sl) {
            if (F::kNibble) {
              uint32_t q[4];
              ldsm4(st_a + sl * 2048 + ((((2 * j + (mi >> 1)) ^ lr) << 4)), q);
              if (FMT == FMT_Q5K || FMT == FMT_Q6K) {  // bits [block][row]: two blocks of rows g and g + 8 a load
                if (FMT == FMT_Q6K ? j % 2 == 0 : j == 0) ldsm4(smem_u32(st) + F::kHighOff + (j + (mi >> 1)) * 2048 + (row0 + 16 * sl + (mi & 1) * 8 + lr) * 16, high[sl]);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
#pragma unroll
                  for (int r = 0; r < 2; ++r) {
                    const uint32_t w = q[2 * k + r], hb = high[sl][2 * (FMT == FMT_Q6K ? j % 2 : j / 2) + r];
                    auto at = [&](int left) { return left > 0 ? hb << left : hb >> -left; };
                    if (FMT == FMT_Q6K) {
                      af[sl][k][r] = ((w << 2) & 0x3C3C3C3Cu) | ((at(6 - 4 * k) & 0xC0C0C0C0u) ^ 0x80808080u);
                      af[sl][k][2 + r] = ((w >> 2) & 0x3C3C3C3Cu) | ((at(4 - 4 * k) & 0xC0C0C0C0u) ^ 0x80808080u);
                    } else {
                      const int f = 2 * (2 * (j % 2) + k);
                      af[sl][k][r] = (w & 0x0F0F0F0Fu) | (at(4 - f) & 0x10101010u);
                      af[sl][k][2 + r] = ((w >> 4) & 0x0F0F0F0Fu) | (at(3 - f) & 0x10101010u);
                    }
                  }
                }
                continue;
              }
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                af[sl][k][0] = q[2 * k] & 0x0F0F0F0Fu;
                af[sl][k][1] = q[2 * k + 1] & 0x0F0F0F0Fu;
                af[sl][k][2] = (q[2 * k] >> 4) & 0x0F0F0F0Fu;
                af[sl][k][3] = (q[2 * k + 1] >> 4) & 0x0F0F0F0Fu;
              }
            } else if (TILED) {
              ldsm4(st_a + sl * 256 + (2 * j) * 4096, af[sl][0]);
              ldsm4(st_a + sl * 256 + (2 * j + 1) * 4096, af[sl][1]);
            } else {
#pragma unroll
              for (int k = 0; k < 2; ++k) ldsm4(st_a + sl * 2048 + (j >> 1) * 16384 + (((2 * ((2 * j + k) & 3) + (mi >> 1)) ^ lr) << 4), af[sl][k]);
            }
          }
        };
        auto frag = [&](int j, int nt) { return *reinterpret_cast<const uint4*>(xf + (j * NT + nt) * 512); };
        // one block's sums into the accumulators: scale and bias of the row, scale and sum of the activations
        auto add = [&](float& ac, const int (&d)[4], int r, float sv, float bv, float xs, float sx) {
          ac = fmaf(sv, digits_sum(d[2 * r], d[2 * r + 1]) * xs, ac);
          if (F::kSums) ac = fmaf(bv, sx, ac);
        };
        auto tab1 = [&](int pr) {  // one row: of pair pr
          if (F::kSums) return *reinterpret_cast<const float2*>(xt + pr * 8);
          return make_float2(*reinterpret_cast<const float*>(xt + pr * 4), 0.f);
        };
        auto tab = [&](int nt, int grp_) {  // scale and sum
          const int at = nt * 4 * F::kGroups + grp_;
          if (F::kSums) return *reinterpret_cast<const float2*>(xt + at * 8);
          return make_float2(*reinterpret_cast<const float*>(xt + at * 4), 0.f);
        };
        if constexpr (FMT == FMT_FP8) {
          // A sum of 128 elements leaves the tensor core, which cuts f32 sums off, before it gets long.  The lane's larger piece is added in one
          // rounding; what that loses goes, with the smaller piece, into a second sum (2-norm of the error against 64 bits, 4096 elements, normal x /
          // of bf16 values: 6.2e-8 / 5.9e-8; both pieces added before they meet the sum 7.3e-8 / 6.3e-8, and with 256 elements in one chain 7.6e-8 /
          // 6.9e-8; the kernel that kept whole rows in tensor memory 6.8e-8 / 7.0e-8; 8192 elements 6.0e-8 / 6.3e-8, and 7.8e-8 / 7.8e-8).
#pragma unroll
          for (int hh = 0; hh < 2; ++hh) {
            float d[SL][NT][4];
#pragma unroll
            for (int sl = 0; sl < SL; ++sl)
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) d[sl][nt][0] = d[sl][nt][1] = d[sl][nt][2] = d[sl][nt][3] = 0.f;
#pragma unroll
            for (int j = 2 * hh; j < 2 * hh + 2; ++j) {
              load_a(j);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                const uint4 b = frag(j, nt);
#pragma unroll
                for (int sl = 0; sl < SL; ++sl) {
                  qmma32(d[sl][nt], af[sl][0], b.x, b.y);
                  qmma32(d[sl][nt], af[sl][1], b.z, b.w);
                }
              }
            }
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              const float xs = *reinterpret_cast<const float*>(xt + nt * 16);
#pragma unroll
              for (int sl = 0; sl < SL; ++sl)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  const float sum = fmaf(d[sl][nt][2 * r], xs, acc[sl][nt][r]), rest = fmaf(d[sl][nt][2 * r + 1], xs, low[sl][nt][r]);
                  low[sl][nt][r] = rest + fmaf(d[sl][nt][2 * r], xs, acc[sl][nt][r] - sum);
                  acc[sl][nt][r] = sum;
                }
            }
          }
        } else if constexpr (FMT == FMT_MLX4) {
          if constexpr (MB == 1) {
#pragma unroll
            for (int jj = 0; jj < 2; ++jj) {
              int d[SL][4];
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const int j = 2 * jj + h;
                load_a(j);
                const uint4 b = frag(j, 0);
#pragma unroll
                for (int sl = 0; sl < SL; ++sl) {
                  int(&e)[4] = d[sl];
                  if (h == 0) imma32<false>(e, af[sl][0][0], af[sl][0][1], af[sl][0][2], af[sl][0][3], b.x, b.y, kAcc0, kAcc0, kAcc0, kAcc0);
                  else imma32<false>(e, af[sl][0][0], af[sl][0][1], af[sl][0][2], af[sl][0][3], b.x, b.y, e[0], e[1], e[2], e[3]);
                  imma32<false>(e, af[sl][1][0], af[sl][1][1], af[sl][1][2], af[sl][1][3], b.z, b.w, e[0], e[1], e[2], e[3]);
                }
              }
              const float2 x = tab1(jj);
#pragma unroll
              for (int sl = 0; sl < SL; ++sl) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  float sv, bv;
                  mlx_scale(sl, r, 2 * jj + half, sv, bv);
                  add(acc[sl][0][r], d[sl], r, sv, bv, x.x, x.y);
                }
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              load_a(j);
              float sv[SL][2], bv[SL][2];
#pragma unroll
              for (int sl = 0; sl < SL; ++sl)
#pragma unroll
                for (int r = 0; r < 2; ++r) mlx_scale(sl, r, j, sv[sl][r], bv[sl][r]);
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                const uint4 b = frag(j, nt);
                const float2 x = tab(nt, j);
#pragma unroll
                for (int sl = 0; sl < SL; ++sl) {
                  int d[4];
                  imma32<false>(d, af[sl][0][0], af[sl][0][1], af[sl][0][2], af[sl][0][3], b.x, b.y, kAcc0, kAcc0, kAcc0, kAcc0);
                  imma32<false>(d, af[sl][1][0], af[sl][1][1], af[sl][1][2], af[sl][1][3], b.z, b.w, d[0], d[1], d[2], d[3]);
#pragma unroll
                  for (int r = 0; r < 2; ++r) add(acc[sl][nt][r], d, r, sv[sl][r], bv[sl][r], x.x, x.y);
                }
              }
            }
          }
        } else if constexpr (FMT == FMT_Q6K) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            load_a(j);
            if constexpr (MB == 1) {
              const uint4 b = frag(j, 0);
              const float2 xx = *reinterpret_cast<const float2*>(xt + j * 8);  // both steps' scales
#pragma unroll
              for (int sl = 0; sl < SL; ++sl) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                  int d[4];
                  imma32<true>(d, af[sl][k][0], af[sl][k][1], af[sl][k][2], af[sl][k][3], k ? b.z : b.x, k ? b.w : b.y, kAcc0, kAcc0, kAcc0, kAcc0);
#pragma unroll
                  for (int r = 0; r < 2; ++r) add(acc[sl][0][r], d, r, rs[sl][r].pair(2 * j + k, half).x, 0.f, k ? xx.y : xx.x, 0.f);
                }
              }
            } else {
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                const int step = 2 * j + k;
                float2 sv[SL][2];
#pragma unroll
                for (int sl = 0; sl < SL; ++sl)
#pragma unroll
                  for (int r = 0; r < 2; ++r) sv[sl][r] = *reinterpret_cast<const float2*>(sc_lane + (16 * sl + 8 * r) * kStagedRow + step * 8);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) {
                  const uint4 b = frag(j, nt);
                  const float2 x = tab(nt, step);
#pragma unroll
                  for (int sl = 0; sl < SL; ++sl) {
                    int d[2][4];
                    imma16(d[0], af[sl][k][0], af[sl][k][1], k ? b.z : b.x, kAcc0);
                    imma16(d[1], af[sl][k][2], af[sl][k][3], k ? b.w : b.y, kAcc0);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                      add(acc[sl][nt][r], d[0], r, sv[sl][r].x, 0.f, x.x, 0.f);
                      add(acc[sl][nt][r], d[1], r, sv[sl][r].y, 0.f, x.x, 0.f);
                    }
                  }
                }
              }
            }
          }
        } else {  // a block per K step
          uint32_t q8[SL][2][4];  // Q8_0: the rows' f16 scales
          if (FMT == FMT_Q80 && MB > 1) {
#pragma unroll
            for (int sl = 0; sl < SL; ++sl)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                const uint4 w = *reinterpret_cast<const uint4*>(meta + (16 * sl + 8 * r) * 16);
                q8[sl][r][0] = w.x;
                q8[sl][r][1] = w.y;
                q8[sl][r][2] = w.z;
                q8[sl][r][3] = w.w;
              }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            load_a(j);
            if constexpr (MB == 1) {
              const uint4 b = frag(j, 0);
              const float2 x = tab1(j);
#pragma unroll
              for (int sl = 0; sl < SL; ++sl) {
                int d[4];
                imma32<F::kSigned>(d, af[sl][0][0], af[sl][0][1], af[sl][0][2], af[sl][0][3], b.x, b.y, kAcc0, kAcc0, kAcc0, kAcc0);
                imma32<F::kSigned>(d, af[sl][1][0], af[sl][1][1], af[sl][1][2], af[sl][1][3], b.z, b.w, d[0], d[1], d[2], d[3]);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  const float2 sb = rs[sl][r].pair(j, half);
                  add(acc[sl][0][r], d, r, sb.x, sb.y, x.x, x.y);
                }
              }
            } else {
              float4 sb[SL][2];  // of the pair's two blocks
#pragma unroll
              for (int sl = 0; sl < SL; ++sl)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                  if (FMT == FMT_Q80) sb[sl][r] = make_float4(f16_lo(q8[sl][r][j]), 0.f, f16_hi(q8[sl][r][j]), 0.f);
                  else sb[sl][r] = *reinterpret_cast<const float4*>(sc_lane + (16 * sl + 8 * r) * kStagedRow + j * 16);
                }
#pragma unroll
              for (int nt = 0; nt < NT; ++nt) {
                const uint4 b = frag(j, nt);
                const float2 x0 = tab(nt, 2 * j), x1 = tab(nt, 2 * j + 1);
#pragma unroll
                for (int sl = 0; sl < SL; ++sl) {
                  int d[2][4];
                  imma32<F::kSigned>(d[0], af[sl][0][0], af[sl][0][1], af[sl][0][2], af[sl][0][3], b.x, b.y, kAcc0, kAcc0, kAcc0, kAcc0);
                  imma32<F::kSigned>(d[1], af[sl][1][0], af[sl][1][1], af[sl][1][2], af[sl][1][3], b.z, b.w, kAcc0, kAcc0, kAcc0, kAcc0);
#pragma unroll
                  for (int r = 0; r < 2; ++r) {
                    add(acc[sl][nt][r], d[0], r, sb[sl][r].x, sb[sl][r].y, x0.x, x0.y);
                    add(acc[sl][nt][r], d[1], r, sb[sl][r].z, sb[sl][r].w, x1.x, x1.y);
                  }
                }
              }
            }
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * rc.s);
        if constexpr (kByChunk) {
#pragma unroll
          for (int sl = 0; sl < SL; ++sl)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
              for (int r = 0; r < 2; ++r) acc[sl][nt][r] += before[sl][nt][r];
        }
      }
      // ---- the item is complete: lanes of a quad meet; lane p of a pair keeps row g + 8 p ----
#pragma unroll
      for (int sl = 0; sl < SL; ++sl) {
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float v0 = acc[sl][nt][0], v1 = acc[sl][nt][1];
          if constexpr (X::kRowTile) {  // all but lane 0's sum meet first, and lanes 0 and 1 have the total: one rounding of its size
            float l0 = low[sl][nt][0], l1 = low[sl][nt][1];
            if (t != 0) {
              l0 = t == 3 ? 0.f : l0 + v0;  // (3: columns without a piece)
              l1 = t == 3 ? 0.f : l1 + v1;
            }
            l0 += __shfl_xor_sync(0xffffffffu, l0, 3);
            l1 += __shfl_xor_sync(0xffffffffu, l1, 3);
            l0 += __shfl_xor_sync(0xffffffffu, l0, 1);
            l1 += __shfl_xor_sync(0xffffffffu, l1, 1);
            v0 = __shfl_sync(0xffffffffu, v0, lane & ~3);
            v1 = __shfl_sync(0xffffffffu, v1, lane & ~3);
            if (!isinf(v0)) v0 += l0;  // (an infinite sum has lost no number)
            if (!isinf(v1)) v1 += l1;
          } else {
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
          }
          float v = p ? v1 : v0;
          if (MB == 1 && !X::kRowTile) v += __shfl_xor_sync(0xffffffffu, v, 2);
          fin[sl * NT + nt] = v;
        }
      }
      if (KG == 1 && !ok) break;
      if constexpr (KG == 2) {
        if (!ok && lane == 0) gave_up[1 + slot] = items + 1;  // (both groups come to the item's meeting, and both leave after it)
        // the groups' sums: the second one's through shared memory (two buffers: the meeting of the next item frees this one)
        float* buf = pair + ((items & 1) * C::kStoring + slot) * (C::kVals * 32) + lane;
        if (grp == 1) {
#pragma unroll
          for (int k = 0; k < C::kVals; ++k) buf[k * 32] = fin[k];
        }
        asm volatile("bar.sync %0, 64;" ::"r"(2 + slot) : "memory");
        if (gave_up[1 + slot] == items + 1) {
          ok = false;
          break;
        }
        if (grp == 1) continue;
#pragma unroll
        for (int k = 0; k < C::kVals; ++k) fin[k] += buf[k * 32];
      }
      if (G) {
        const int row = sw.tile * kTileRows + row0 + g + 8 * p, out_dim = a.seg[0].out_dim;  // of the first slab
        float* const out = a.seg[0].out;
        if (sw.entry != cur_entry) {
          cur_entry = sw.entry;
          nb = __ldg(&entry_at(cur_entry)->count);
        }
        if (kWork && a.gdirect == 2 && sw.mat == 0) {
#pragma unroll
          for (int k = 0; k < C::kVals; ++k) gate[kWork ? k : 0] = fin[k];
          continue;
        }
#pragma unroll
        for (int k = 0; k < C::kVals; ++k) {
          const int m = act(k), r = row + 16 * (k / NT);
          if (m >= nb) continue;
          if constexpr (kWork) {
            const MmaWorkEntry* we = reinterpret_cast<const MmaWorkEntry*>(a.gwork) + cur_entry;
            if (a.gdirect == 2) {
              out[(size_t)__ldg(&we->g.item[m]) * out_dim + r] = gelu_tanh(gate[k]) * fin[k];
            } else {
              float* dst = reinterpret_cast<float*>(__ldg(reinterpret_cast<const unsigned long long*>(&we->dst[m])));
              if (r < __ldg(&we->room[m])) atomicAdd(dst + r, fin[k] * __ldg(&we->weight[m]));  // items may share a destination row
            }
          } else {
            const int orow = a.gdirect ? __ldg(&entry_at(cur_entry)->item[m]) : cur_entry * MB + m;
            out[(size_t)orow * out_dim + sw.mat * (a.gtpe * kTileRows) + r] = fin[k];
          }
        }
      } else if (a.cluster) {
        have = true;
        break;  // the CTA's one item: below
      } else if (a.splits == 1) {
        store(sw.tile, items, [&](int k) { return fin[k]; });
      } else {
        // Partial sums of this K range go to scratch; the warp that arrives last at its rows of the tile adds the
        // partials in split order (so the result does not depend on arrival order) and stores.
        constexpr int kPart = C::kVals * 32;
        float* part = a.scratch + (((size_t)sw.tile * a.splits + sw.split) * C::kStoring + slot) * kPart + lane;
#pragma unroll
        for (int k = 0; k < C::kVals; ++k) part[k * 32] = fin[k];
        __threadfence();
        __syncwarp();
        unsigned int n = 0;
        if (lane == 0) n = atomicAdd(a.counters + sw.tile * kConsumers + slot, 1u);
        n = __shfl_sync(0xffffffffu, n, 0);
        if (n == (unsigned)a.splits - 1) {
          __threadfence();
          const float* base = a.scratch + ((size_t)sw.tile * a.splits * C::kStoring + slot) * kPart + lane;
          store(sw.tile, items, [&](int k) {
            float sum = 0.f;
            for (int s2 = 0; s2 < a.splits; ++s2) sum += __ldcg(base + (size_t)s2 * (C::kStoring * kPart) + k * 32);
            return sum;
          });
          if (lane == 0) a.counters[sw.tile * kConsumers + slot] = 0;
        }
      }
    }
    if (!ok && lane == 0) *gave_up = 1;
    if (a.cluster) {
      // The K splits of this tile are the CTAs of this cluster (rank == split) and each has this one item.  Ranks above 0
      // put their sums into rank 0's shared memory; rank 0 adds them in split order, the order of the scratch path.
      __syncwarp();
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
      if (have && sw.split != 0) {
        const uint32_t dst = cluster_map(smem_u32(recv + (size_t)(sw.split - 1) * (C::kRecv / 4) + slot * (C::kVals * 32) + lane), 0);
#pragma unroll
        for (int k = 0; k < C::kVals; ++k) cluster_store_f32(dst + k * 128, fin[k]);
      }
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      if (sw.split == 0) {
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (have) {
          store(sw.tile, 0, [&](int k) {
            float sum = fin[k];
            for (int s2 = 1; s2 < a.splits; ++s2) sum += recv[(size_t)(s2 - 1) * (C::kRecv / 4) + slot * (C::kVals * 32) + k * 32 + lane];
            return sum;
          });
        }
      }
    }
  }
  if (a.cluster && warp == kConsumers) {
    __syncwarp();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (blockIdx.x % a.splits == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  // ---- wind down: outstanding copies are drained ----
  __syncthreads();
  if constexpr (kPlain) {
    if (__builtin_expect(__any_sync(0xffffffffu, odd != 0 && a.plain), 0)) {
      StageWalk again(a);
      for (int item = 0; again.live(a); again.next_item(a), ++item) {
        if (!__any_sync(0xffffffffu, (odd >> (item < 31 ? item : 31)) & 1u)) continue;
        const int sg = seg_of(again.tile), slot = C::KG == 2 ? warp & 3 : warp;
        store_again<FMT, MB, TILED, C::kVals>(a, sg, (again.tile - a.seg[sg].tile0) * kTileRows + slot * (16 * SL) + (lane >> 2) + 8 * (lane & 1), lane);
      }
    }
  }
  if (*gave_up && warp == kConsumers && lane == 0) {
    // a waiter gave up: copies may still be in flight; give each ring slot a bounded chance to land
    for (int s = 0; s < S; ++s) {
      long long t0 = clock64();
      while (!mbar_try_wait(full0 + 8 * s, 0) && !mbar_try_wait(full0 + 8 * s, 1) && clock64() - t0 < kTimeoutCycles / 8) {
      }
    }
  }
}

// ---- host side --------------------------------------------------------------------------

// Row-major words + {scale,bias} table -> tiled blocks; one thread per 16-byte unit / meta row.
__global__ void mlx_tile_kernel(const uint32_t* __restrict__ qw, const uint32_t* __restrict__ sb,
                                unsigned char* __restrict__ tiled, int out_dim, int in_dim, int ntiles, int nchunks) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t nblocks = (size_t)ntiles * nchunks;
  if (idx >= nblocks * (128 * 9)) return;
  size_t blk = idx / (128 * 9);
  int rem = (int)(idx - blk * (128 * 9));
  int tile = (int)(blk / nchunks), chunk = (int)(blk - (size_t)tile * nchunks);
  int r = rem / 9, u = rem - r * 9;
  int row = tile * 128 + r;
  uint4 v = make_uint4(0, 0, 0, 0);
  unsigned char* dst = tiled + blk * Fmt<FMT_MLX4>::kStageBytes;
  if (u < 8) {
    if (row < out_dim) v = *reinterpret_cast<const uint4*>(qw + (size_t)row * (in_dim / 8) + chunk * 32 + u * 4);
    *reinterpret_cast<uint4*>(dst + r * 128 + ((u ^ (r & 7)) << 4)) = v;
  } else {
    if (row < out_dim) v = *reinterpret_cast<const uint4*>(sb + (size_t)row * (in_dim / 64) + chunk * 4);
    *reinterpret_cast<uint4*>(dst + Fmt<FMT_MLX4>::kStageWBytes + r * 16) = v;
  }
}

bool mlx_mma_supported(const goph_mlx_weight* w) {
  return w->sb_bf16 && w->group_size == 64 && w->in_dim % kChunkK == 0 && w->in_dim <= 65536;
}

int mlx_mma_make_tiled(goph_mlx_weight* w) {
  int ntiles = (w->out_dim + kTileRows - 1) / kTileRows, nchunks = w->in_dim / kChunkK;
  size_t bytes = (size_t)ntiles * nchunks * Fmt<FMT_MLX4>::kStageBytes;
  unsigned char* t = nullptr;
  GOPH_CUDA(cudaMalloc(&t, bytes));
  size_t threads = (size_t)ntiles * nchunks * 128 * 9;
  mlx_tile_kernel<<<(unsigned)((threads + 255) / 256), 256>>>(w->qweight, reinterpret_cast<const uint32_t*>(w->sb), t,
                                                              w->out_dim, w->in_dim, ntiles, nchunks);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaFree(t);
    return fail_cuda(e, "mlx_tile_kernel");
  }
  w->tiled = t;
  w->bytes = bytes;
  return GOPH_OK;
}

struct MmaDeviceBufs {
  unsigned char* xb = nullptr;  // prepared activations of the launch in flight
  int* status = nullptr;
  float* scratch = nullptr;
  unsigned int* counters = nullptr;
};
// Fixed-size device scratch of the split-K fix-up: at most 2 x 160 items of 128 rows x 8
// activation rows, plus a counter per tile and warp.  Allocated once per device.
constexpr size_t kScratchFloats = (size_t)2 * 160 * kTileRows * 8;
constexpr size_t kMaxCounters = 4096 * kConsumers;
// Prepared activations: up to 8 rows of up to 65536 elements.
constexpr int kMaxPrepIn = 65536;  // mlx_mma_supported's bound on in_dim
constexpr size_t kPrepXbBytes = (size_t)(kMaxPrepIn / kChunkK) * XBlock<FMT_Q4K, 8>::kBytes;
static_assert(XBlock<FMT_FP8, 4>::kBytes <= XBlock<FMT_Q4K, 8>::kBytes, "the widest activations");

// The buffers of a device are allocated on first use.  Nothing is published until every
// allocation has succeeded (a failure frees what it got and the next call tries again), and
// first calls from several threads are serialised.
static MmaDeviceBufs* device_bufs(int device) {
  static MmaDeviceBufs bufs[kMaxDevices];
  static bool ready[kMaxDevices] = {};
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (ready[device]) return &bufs[device];
  MmaDeviceBufs b;
  bool ok = cudaMalloc(&b.status, sizeof(int)) == cudaSuccess &&
            cudaMalloc(&b.scratch, kScratchFloats * sizeof(float)) == cudaSuccess &&
            cudaMalloc(&b.counters, kMaxCounters * sizeof(unsigned int)) == cudaSuccess &&
            cudaMalloc(&b.xb, kPrepXbBytes) == cudaSuccess;
  ok = ok && cudaMemset(b.xb, 0, kPrepXbBytes) == cudaSuccess && cudaMemset(b.status, 0, sizeof(int)) == cudaSuccess &&
       cudaMemset(b.counters, 0, kMaxCounters * sizeof(unsigned int)) == cudaSuccess &&
       cudaDeviceSynchronize() == cudaSuccess;
  if (!ok) {
    cudaGetLastError();
    cudaFree(b.status);
    cudaFree(b.scratch);
    cudaFree(b.counters);
    cudaFree(b.xb);
    return nullptr;
  }
  bufs[device] = b;
  ready[device] = true;
  return &bufs[device];
}

void mlx_mma_status_clear(int device) {
  MmaDeviceBufs* b = device_bufs(device);
  if (b) cudaMemset(b->status, 0, sizeof(int));
}

int mlx_mma_status(int device) {
  MmaDeviceBufs* b = device_bufs(device);
  int v = -1;
  if (b) cudaMemcpy(&v, b->status, sizeof(int), cudaMemcpyDeviceToHost);
  return v;
}

// Weights of one launch that share x, as the launch code sees them.
struct RowWeights {
  int device, in_dim, n;
  RowSeg seg[kMaxRowSeg];              // tile0 filled in
  const QMaps* maps[kMaxRowSeg] = {};  // row-major
  bool unordered = false;              // callers need no order between such products: no scratch of the device's (unless an output meets x)
  size_t scratch_bytes = kScratchFloats * sizeof(float), counters = kMaxCounters;
};

// Shared memory of a CTA: half of an SM's, so that two CTAs share one (the next launch's first stages are under way while
// this one ends), or all of it where the activations do not leave the ring its stages.
constexpr size_t kHalfSmem = 113 * 1024, kWholeSmem = 222 * 1024;

// Clusters of `splits` CTAs that the device holds at once, one or two CTAs to an SM (a property of how the SMs are grouped:
// every instantiation has the same threads and registers); asked once per device.
static int cluster_room(int device, int splits, bool whole) {
  static std::mutex mu;
  static int room[kMaxDevices][2][kMaxSplits + 1];
  static bool known[kMaxDevices] = {};
  std::lock_guard<std::mutex> lock(mu);
  if (!known[device]) {
    auto kern = mlx_mma_kernel<FMT_MLX4, 1, true>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWholeSmem);
    cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    for (int w = 0; w < 2; ++w) {
      for (int n = 2; n <= kMaxSplits; ++n) {
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = n;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof cfg);
        cfg.gridDim = dim3(n * 64);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = w ? kWholeSmem : kHalfSmem;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&room[device][w][n], kern, &cfg) != cudaSuccess) {
          cudaGetLastError();
          room[device][w][n] = 0;
        }
      }
    }
    known[device] = true;
  }
  return room[device][whole][splits];
}

// How a product is cut up and who prepares its activations.
struct RowPlan {
  bool own, whole;  // by the product's CTAs themselves, each for its K range; one CTA to an SM
  int splits;
  bool cluster;
};

template <int FMT, int MB, bool FUSED, bool TILED>
static int launch_impl(const RowWeights& w, MmaArgs a, cudaStream_t stream, SharedX* xs, const RowPlan& plan) {
  typedef RowSmem<FMT, MB, FUSED, false, TILED> M;
  const int splits = plan.splits;
  a.splits = splits;
  a.items = a.ntiles * splits;
  a.cmax = (a.nchunks + splits - 1) / splits;
  a.cluster = plan.cluster;
  const int recv = plan.cluster ? splits - 1 : 0;
  a.stages = M::stages(plan.whole ? kWholeSmem : kHalfSmem, a.cmax, recv);
  size_t smem = M::bytes(a.stages, a.cmax, recv);
  if (plan.whole && smem <= kHalfSmem) smem = kHalfSmem + 1024;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (!FUSED && !xs->prepared) {
    // activations -> digits, sums and scales, once per launch
    cfg.gridDim = dim3(a.batch * a.nchunks);
    cfg.blockDim = dim3(FMT == FMT_FP8 ? 32 : 128);
    note_launch();
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, mlx_prep_x_kernel<FMT, MB>, a.x, const_cast<unsigned char*>(a.xb), a.in_dim, a.digits));
    xs->prepared = true;
  }
  auto kern = mlx_mma_kernel<FMT, MB, FUSED, false, TILED>;
  static bool sized[kMaxDevices] = {};
  if (!sized[w.device]) {
    GOPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWholeSmem));
    GOPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    sized[w.device] = true;
  }
  const int slots = device_state(w.device).sm_count * (plan.whole ? 1 : 2);
  int grid = plan.cluster || a.items < slots ? a.items : slots;  // (a CTA of a cluster has one item)
  // FUSED: a CTA prepares the activations of one K range, so all its items must be of one split:
  // item w is split w % splits, and a grid that is a multiple of the splits keeps that fixed per CTA
  if (FUSED && a.items > grid) grid -= grid % splits;
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  if (plan.cluster) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  // GOPH_TRACE_LAUNCH=1 in the environment: one line per tensor-core product with its launch plan
  static const bool trace = getenv("GOPH_TRACE_LAUNCH") != nullptr;
  if (trace)
    fprintf(stderr, "goph: mlx_mma_kernel fmt=%d tiled=%d weights=%d out=%d in=%d rows=%d grid=%d splits=%d stages=%d fused=%d cluster=%d smem=%d\n", FMT, (int)TILED, a.nseg,
            a.seg[0].out_dim, a.in_dim, a.batch, grid, splits, a.stages, (int)FUSED, a.cluster, (int)smem);
  note_launch();
  if constexpr (TILED) {
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, kern, a, NoMaps()));
  } else {
    RowMaps maps;
    for (int i = 0; i < w.n; ++i) memcpy(maps.map[i], w.maps[i]->map, sizeof maps.map[i]);
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, kern, a, maps));
  }
  return GOPH_OK;
}

// 0: done; 1: the activations of so many rows do not fit (nothing launched); else an error.
constexpr int kDoesNotFit = 1 << 20;
template <int FMT, int MB, bool TILED>
static int launch_one(const RowWeights& w, const MmaArgs& a, cudaStream_t stream, SharedX* xs) {
  constexpr bool kBytes = !Fmt<FMT>::kNibble;
  typedef RowSmem<FMT, MB, true, false, TILED> Own;
  typedef RowSmem<FMT, MB, false, false> Front;
  const int sms = device_state(w.device).sm_count, tiles = a.ntiles;
  // No scratch: activations by the CTAs, sums inside clusters.  (An output that meets x has x prepared in front all the same, in the device's scratch.)
  const bool alone = (w.unordered && !xs->written) || !TILED;
  RowPlan p;
  // The lines (B200, us a call, weights from HBM).  A CTA to an SM, with a ring of all that is left: products that are over in a few stages (one row, MLX4
  // 4096x4096 4.4, two to an SM 4.6; 14336x4096 8.3 / 7.7), and several rows, whose activations leave half an SM too little (four rows 14336x4096 10.8 / 11.4;
  // two of Q8_0 12.2 / 12.9).  By the CTAs themselves or in front: one row 4096x4096 4.4 / 6.2, 28672x4096 13.0 / 12.9,
  // 28672x8192 24.5 / 22.5; two rows 4096x4096 4.6 / 6.9, 14336x4096 8.7 / 9.6, where nothing is cut 28672x4096 15.5 / 13.5 (Q8_0 22.6 / 21.3); four 4096x4096 6.1 / 6.3,
  // 14336x4096 14.3 / 10.8.  Up to 17 chunks a CTA (two a warp) are its own.  MLX products of more than a tile for two SMs, fewer than one for each, and more than 17 chunks
  // have theirs in front: 14000x4608 one row 9.1 / 9.4, two rows 14336x4096 8.7 / 9.6 (a call of several such weights prepares them once).
  const bool small = (long)tiles * a.nchunks <= 8l * sms;
  p.whole = small || MB == 8 || (MB == 4 && (FMT != FMT_MLX4 || tiles < sms)) || (MB == 2 && kBytes && tiles < sms);
  const int most = 1 + 28 * 1024 / RowCfg<FMT, MB, false>::kRecv;  // (of the others' sums that the first CTA of a cluster has room for)
  auto cut = [&](bool whole) {
    const int slots = sms * (whole ? 1 : 2);
    int n = slots / tiles;
    if (n > a.nchunks) n = a.nchunks;
    if (n > kMaxSplits) n = kMaxSplits;
    if (n > most) n = most;
    if (n > 8 && 16 * tiles > slots) n = 8;  // (larger clusters where eight CTAs a tile leave more than half of the places empty: 256x16384 5.7 / 4.5; 4096x14336 8.4 / 9.2)
    const bool clusters = options().mlx_cluster || alone;
    if (!whole && n == 8 && 40 * tiles > 4 * slots) n = 7;  // (eights pack badly where they would have to fill the device, 30 tiles to 37: MLX4 4096x14336 9.2 / 8.3)
    if (clusters)
      while (n > 1 && cluster_room(w.device, n, whole) < tiles) --n;
    if (options().mlx_splits > 0 && !alone) n = options().mlx_splits < a.nchunks ? options().mlx_splits : a.nchunks;
    while (n > 1 && ((size_t)tiles * n * RowCfg<FMT, MB, false>::kRecv > w.scratch_bytes || (size_t)tiles * kConsumers > w.counters)) --n;
    p.whole = whole;
    p.splits = n < 1 ? 1 : n;
    p.cluster = clusters && n > 1 && n <= most && n <= kMaxSplits && (long)tiles * n <= slots && cluster_room(w.device, n, whole) >= tiles;
  };
  cut(p.whole);
  const int cmax = (a.nchunks + p.splits - 1) / p.splits;
  if (MB == 1) p.own = p.splits > 1 || a.nchunks <= 24;
  else if (MB == 2) p.own = small || (p.splits > 1 ? !kBytes : kBytes);
  else p.own = false;
  if (a.batch * cmax <= 17) p.own = true;
  if (FMT == FMT_MLX4 && 2 * tiles > sms && tiles < sms && a.batch * a.nchunks > 17) p.own = false;
  if (!options().mlx_fuse || xs->written || p.splits > sms) p.own = false;
  if (alone) p.own = true;
  // a ring of three stages at least (of two where groups of warps take turns): else a whole SM, else a launch in front
  for (int t = 0; t < 5; ++t) {
    const int recv = p.cluster ? p.splits - 1 : 0, range = (a.nchunks + p.splits - 1) / p.splits, least = RowCfg<FMT, MB, false>::KG == 2 && p.whole ? 2 : 3;
    const size_t budget = p.whole ? kWholeSmem : kHalfSmem;
    if (p.own && Own::stages(budget, range, recv) >= least) return launch_impl<FMT, MB, true, TILED>(w, a, stream, xs, p);
    if constexpr (TILED)
      if (!p.own && Front::stages(budget, range, recv) >= least) return launch_impl<FMT, MB, false, true>(w, a, stream, xs, p);
    if (!p.whole) {
      cut(true);
    } else if (alone) {
      // K ranges short enough for a CTA's activations, in more clusters than the device holds at once: they run in waves (9473 rows and
      // more of 14593 elements and more).  The cut whose waves take the fewest chunks, a start of four chunks for each.  B200, us a call, one row, CUDA cores / so:
      // Q8_0 9600x14624 63.5 / 41.0, FP8 9600x15696 53.2 / 46.0, MLX 9600x20800 67.6 / 44.0.
      long best = 0;
      for (int n = p.splits + 1; n <= kMaxSplits && n <= most && n <= a.nchunks; ++n) {
        const int room = cluster_room(w.device, n, true), range = (a.nchunks + n - 1) / n;
        if (room == 0 || Own::stages(kWholeSmem, range, n - 1) < least) continue;
        const long cost = (long)((tiles + room - 1) / room) * (range + 4);
        if (best && cost >= best) continue;
        best = cost;
        p.splits = n;
      }
      if (!best) break;
      p.cluster = true;
    } else if (p.own) {
      p.own = false;
    } else if (p.cluster) {
      p.cluster = false;  // (the sums meet in scratch and need no shared memory)
    } else {
      break;
    }
  }
  return kDoesNotFit;
}

// The next rows of a call: as many as fit a launch.  Their number, or minus the error.
template <int FMT, bool TILED>
static int rows_slice(const RowWeights& w0, MmaArgs a, cudaStream_t stream, SharedX* xs, int* taken = nullptr) {
  RowWeights w = w0;
  a.in_dim = w.in_dim;
  a.nchunks = (w.in_dim + kChunkK - 1) / kChunkK;
  a.nseg = w.n;
  a.ntiles = 0;
  for (int i = 0; i < w.n; ++i) {
    a.seg[i] = w.seg[i];
    a.seg[i].tile0 = a.ntiles;
    a.ntiles += (w.seg[i].out_dim + kTileRows - 1) / kTileRows;
  }
  constexpr int kMost = FMT == FMT_FP8 ? 4 : 8;
  for (int nb = a.batch < kMost ? a.batch : kMost; nb > 0; nb = nb > 4 ? 4 : nb > 2 ? 2 : nb - 1) {
    a.batch = nb;
    const int rc = nb == 1 ? launch_one<FMT, 1, TILED>(w, a, stream, xs) : nb == 2 ? launch_one<FMT, 2, TILED>(w, a, stream, xs)
                 : nb <= 4 ? launch_one<FMT, 4, TILED>(w, a, stream, xs) : launch_one<FMT, kMost, TILED>(w, a, stream, xs);
    if (rc == kDoesNotFit) continue;
    if (taken) *taken = nb;
    return rc;
  }
  return fail(GOPH_E_UNSUPPORTED, "tensor-core path: activations of %d elements leave no room for the ring", w.in_dim);
}

template <int FMT, bool TILED>
static int rows_launch(const RowWeights& w0, const float* x, int batch, int digits, cudaStream_t stream, SharedX* shared) {
  MmaDeviceBufs* bufs = device_bufs(w0.device);
  if (!bufs) return fail(GOPH_E_NOMEM, "cannot allocate the tensor-core path's device scratch");
  RowWeights w = w0;
  MmaArgs a;
  memset(&a, 0, sizeof a);
  a.status = bufs->status;
  a.scratch = bufs->scratch;
  a.counters = bufs->counters;
  a.xb = bufs->xb;
  a.digits = digits == 3 ? 3 : 4;
  bool written = shared && shared->written;
  if (!shared)
    for (int i = 0; i < w.n; ++i) written = written || floats_meet(w.seg[i].out, (uint64_t)batch * w.seg[i].out_dim, x, (uint64_t)batch * w.in_dim);
  a.plain = !written && (FMT == FMT_FP8 || w.unordered || batch > 4);
  for (int b0 = 0; b0 < batch;) {
    a.x = x + (size_t)b0 * w.in_dim;
    for (int i = 0; i < w.n; ++i) w.seg[i].out = w0.seg[i].out + (size_t)b0 * w.seg[i].out_dim;
    a.batch = batch - b0;
    SharedX own;  // (rows of a later launch of this call do not have the scratch's activations)
    own.written = written;
    int taken = 0;
    if (int rc = rows_slice<FMT, TILED>(w, a, stream, shared && batch <= 8 ? shared : &own, &taken)) return rc;
    b0 += taken;
  }
  return GOPH_OK;
}

int mlx_mma_launch(const goph_mlx_weight* w, float* out, const float* x, int batch, int digits, cudaStream_t stream,
                   SharedX* shared) {
  if (!w->tiled) return fail(GOPH_E_UNSUPPORTED, "weight is not in the tiled layout");
  RowWeights d;
  d.device = w->device;
  d.in_dim = w->in_dim;
  d.n = 1;
  d.seg[0] = RowSeg{w->tiled, out, w->out_dim, 0};
  return rows_launch<FMT_MLX4, true>(d, x, batch, digits, stream, shared);
}

int fp8_mma_launch_rows(const goph_fp8_linear* w, float* out, const float* x, int batch, cudaStream_t stream) {
  RowWeights d;
  d.device = w->device;
  d.in_dim = w->in_dim;
  d.n = 1;
  d.seg[0] = RowSeg{w->tiled ? w->tiled : w->weight, out, w->out_dim, 0, w->scale, w->bias};
  d.maps[0] = &w->qmaps;
  return w->tiled ? rows_launch<FMT_FP8, true>(d, x, batch, 4, stream, nullptr) : rows_launch<FMT_FP8, false>(d, x, batch, 4, stream, nullptr);
}

bool mlx_mma_ready(int device) { return device_bufs(device) != nullptr; }

int mlx_mma_launch_rows(int n, const goph_mlx_weight* const* ws, float* const* outs, const float* x, int batch, int digits, cudaStream_t stream) {
  for (int i0 = 0; i0 < n; i0 += kMaxRowSeg) {
    RowWeights d;
    d.device = ws[0]->device;
    d.in_dim = ws[0]->in_dim;
    d.n = n - i0 < kMaxRowSeg ? n - i0 : kMaxRowSeg;
    for (int i = 0; i < d.n; ++i) {
      const goph_mlx_weight* w = ws[i0 + i];
      d.seg[i] = RowSeg{nullptr, outs[i0 + i], w->out_dim, 0};
      d.maps[i] = &w->qmaps;
    }
    if (int rc = rows_launch<FMT_MLX4, false>(d, x, batch, digits, stream, nullptr)) return rc;
  }
  return GOPH_OK;
}

// ---- grouped launches (mixture-of-experts) -----------------------------------------------------

// The activations of every (entry, row) as the tensor core wants them: block = one row of one entry,
// a warp takes chunks; arithmetic and layout are mlx_prep_x_kernel's.  PHASE 0: the row is
// the item's token in src[tokens][in_dim]; PHASE 1: silu(g) * u of the gate and up results
// src[entry * MB + m][2][in_dim] (kernels.SiLU then the multiply, backends/simd/kernels/activation.go:15-24;
// single-precision exp as in the CUDA-core expert kernels).
template <int MB, int PHASE>
__global__ void __launch_bounds__(256)
moe_mma_prep_kernel(const MmaGroupEntry* __restrict__ work, const int* __restrict__ count, int max_entries,
                    const float* __restrict__ src, int in_dim, int top_k, unsigned char* __restrict__ xb, size_t xb_stride) {
  pdl_launch_dependents();
  pdl_wait();
  const int entry = blockIdx.x / MB, m = blockIdx.x - entry * MB;
  int live = __ldcg(count);
  if (live > max_entries) live = max_entries;
  if (entry >= live) return;
  const MmaGroupEntry* ge = work + entry;
  if (m >= ge->count) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* row = PHASE == 0 ? src + (size_t)(ge->item[m] / top_k) * in_dim : src + (size_t)(entry * MB + m) * 2 * in_dim;
  unsigned char* bdst = xb + (size_t)entry * xb_stride;
  for (int c = warp; c < in_dim / kChunkK; c += 8) {
    const int k = c * kChunkK + lane * 8;
    float v[8];
    load_eight(row + k, v);
    if (PHASE == 1) {
      float u[8];
      load_eight(row + in_dim + k, u);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = __fmul_rn(__fdiv_rn(v[i], __fadd_rn(1.0f, expf(-v[i]))), u[i]);
    }
    prep_chunk<FMT_MLX4, MB>(v, lane, bdst + (size_t)c * XBlock<FMT_MLX4, MB>::kBytes, m, 4);
  }
}

bool mlx_mma_grouped_supported(int hidden, int inter) {
  return hidden % kChunkK == 0 && inter % kChunkK == 0 && hidden % kTileRows == 0 && inter % kTileRows == 0 && hidden <= 16384 &&
         inter <= 16384;
}
size_t mlx_mma_grouped_xb_bytes(int in_dim, int rows) {
  return (size_t)(in_dim / kChunkK) * (rows == 2 ? XBlock<FMT_MLX4, 2>::kBytes : XBlock<FMT_MLX4, 4>::kBytes);
}

template <int MB>
static int launch_grouped(int device, const MmaGroupLaunch& g, cudaStream_t stream) {
  typedef RowSmem<FMT_MLX4, MB, false, true> M;
  MmaDeviceBufs* bufs = device_bufs(device);
  if (!bufs) return fail(GOPH_E_NOMEM, "cannot allocate the tensor-core path's device scratch");
  DeviceState& st = device_state(device);
  MmaArgs a;
  memset(&a, 0, sizeof a);
  a.status = bufs->status;
  a.xb = g.xb;
  a.nseg = 1;
  a.seg[0].out = g.out;
  a.seg[0].out_dim = g.mats * g.rows;
  a.in_dim = g.in_dim;
  a.batch = MB;
  a.digits = 4;
  a.ntiles = g.rows / kTileRows;
  a.nchunks = g.in_dim / kChunkK;
  a.splits = 1;
  a.items = g.max_entries * g.mats * a.ntiles;
  a.gwork = g.work;
  a.gcount = g.count;
  a.gmax = g.max_entries;
  a.gtpe = a.ntiles;
  a.gmats = g.mats;
  a.gfirst = g.first;
  a.gdirect = g.phase == 1;
  a.gxb = mlx_mma_grouped_xb_bytes(g.in_dim, MB);
  a.stages = M::stages(kHalfSmem, 0, 0);
  const size_t smem = M::bytes(a.stages, 0, 0);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(g.max_entries * MB);
  cfg.blockDim = dim3(256);
  note_launch();
  if (g.phase == 0)
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, moe_mma_prep_kernel<MB, 0>, g.work, g.count, g.max_entries, g.src, g.in_dim, g.top_k, g.xb, a.gxb));
  else
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, moe_mma_prep_kernel<MB, 1>, g.work, g.count, g.max_entries, g.src, g.in_dim, g.top_k, g.xb, a.gxb));
  auto kern = mlx_mma_kernel<FMT_MLX4, MB, false, true>;
  GOPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cfg.gridDim = dim3(a.items < 2 * st.sm_count ? a.items : 2 * st.sm_count);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  note_launch();
  GOPH_CUDA(cudaLaunchKernelEx(&cfg, kern, a, NoMaps()));
  return GOPH_OK;
}

int mlx_mma_launch_grouped(int device, const MmaGroupLaunch& g, cudaStream_t stream) {
  if (g.entry_rows == 2) return launch_grouped<2>(device, g, stream);
  if (g.entry_rows == 4) return launch_grouped<4>(device, g, stream);
  return fail(GOPH_E_INVALID, "grouped launch: entries of %d items", g.entry_rows);
}

// ---- GGUF Q4_K / Q8_0 in the tiled layouts ------------------------------------------------------

// Device super-blocks {16-byte header, 8 x 16 bytes of nibbles} -> tiled stages; one thread per 16-byte unit.
__global__ void q4k_tile_kernel(const unsigned char* __restrict__ blocks, unsigned char* __restrict__ tiled, int out_dim,
                                int ntiles, int nchunks) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t nstages = (size_t)ntiles * nchunks;
  if (idx >= nstages * (128 * 9)) return;
  size_t stg = idx / (128 * 9);
  int rem = (int)(idx - stg * (128 * 9));
  int tile = (int)(stg / nchunks), chunk = (int)(stg - (size_t)tile * nchunks);
  int r = rem / 9, u = rem - r * 9;
  int row = tile * 128 + r;
  uint4 v = make_uint4(0, 0, 0, 0);
  unsigned char* dst = tiled + stg * Fmt<FMT_Q4K>::kStageBytes;
  const unsigned char* src = blocks + ((size_t)row * nchunks + chunk) * 144;
  if (u < 8) {
    if (row < out_dim) v = *reinterpret_cast<const uint4*>(src + 16 + 16 * u);
    *reinterpret_cast<uint4*>(dst + r * 128 + ((u ^ (r & 7)) << 4)) = v;
  } else {
    if (row < out_dim) v = *reinterpret_cast<const uint4*>(src);
    *reinterpret_cast<uint4*>(dst + Fmt<FMT_Q4K>::kStageWBytes + r * 16) = v;
  }
}

// Byte plane (q + 128) and f16 scales -> tiled stages of signed bytes; one thread per 16-byte half block.
__global__ void q80_tile_kernel(const unsigned char* __restrict__ plane, const uint16_t* __restrict__ d16,
                                unsigned char* __restrict__ tiled, int out_dim, int in_dim, int ntiles, int nchunks) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t nstages = (size_t)ntiles * nchunks;
  if (idx >= nstages * (128 * 16)) return;
  size_t stg = idx / (128 * 16);
  int rem = (int)(idx - stg * (128 * 16));
  int tile = (int)(stg / nchunks), chunk = (int)(stg - (size_t)tile * nchunks);
  int r = rem >> 4, hb = rem & 15, step = hb >> 1, half = hb & 1;
  int row = tile * 128 + r;
  unsigned char* dst = tiled + stg * Fmt<FMT_Q80>::kStageBytes;
  uint4 v = make_uint4(0, 0, 0, 0);
  const bool in = row < out_dim && chunk * 256 + step * 32 < in_dim;  // (rows may end inside a chunk, at a block)
  if (in) {
    v = *reinterpret_cast<const uint4*>(plane + (size_t)row * in_dim + chunk * 256 + step * 32 + half * 16);
    v.x ^= 0x80808080u;
    v.y ^= 0x80808080u;
    v.z ^= 0x80808080u;
    v.w ^= 0x80808080u;
  }
  *reinterpret_cast<uint4*>(dst + step * 4096 + half * 2048 + (r >> 3) * 128 + (r & 7) * 16) = v;
  if (half == 0) {
    uint16_t d = in ? d16[(size_t)row * (in_dim / 32) + chunk * 8 + step] : (uint16_t)0;
    *reinterpret_cast<uint16_t*>(dst + Fmt<FMT_Q80>::kStageWBytes + r * 16 + step * 2) = d;
  }
}

// dequantRowQ4KTo / dequantRowQ8_0To from the tiled layouts (loader/gguf/quant_matrix.go:138-158, :281-329).
__global__ void q4k_dequant_tiled_kernel(const unsigned char* __restrict__ tiled, float* __restrict__ out, int out_dim,
                                         int in_dim, int nchunks) {
  size_t u = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // 32-element unit of the row-major result
  size_t units_per_row = in_dim / 32;
  if (u >= (size_t)out_dim * units_per_row) return;
  int row = (int)(u / units_per_row), unit = (int)(u - (size_t)row * units_per_row);
  int chunk = unit >> 3, sblk = unit & 7, r = row & 127;
  const unsigned char* stg = tiled + ((size_t)(row >> 7) * nchunks + chunk) * Fmt<FMT_Q4K>::kStageBytes;
  uint4 h = *reinterpret_cast<const uint4*>(stg + Fmt<FMT_Q4K>::kStageWBytes + r * 16);
  uint4 q = *reinterpret_cast<const uint4*>(stg + r * 128 + ((sblk ^ (r & 7)) << 4));
  int bit = 12 * sblk, wi = bit >> 5, sh = bit & 31;
  uint32_t lo = wi == 0 ? h.y : wi == 1 ? h.z : h.w, hi = wi == 0 ? h.z : wi == 1 ? h.w : 0u;
  uint32_t f = __funnelshift_r(lo, hi, sh) & 0xFFFu;
  float sd = __fmul_rn((float)(f & 63u), __half2float(__ushort_as_half((unsigned short)(h.x & 0xFFFFu))));
  float md = __fmul_rn((float)(f >> 6), __half2float(__ushort_as_half((unsigned short)(h.x >> 16))));
  float4* o = reinterpret_cast<float4*>(out + u * 32);
  uint32_t ws[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = __fsub_rn(__fmul_rn(sd, (float)((ws[k] >> (4 * e)) & 0xF)), md);
    o[2 * k] = make_float4(v[0], v[1], v[2], v[3]);
    o[2 * k + 1] = make_float4(v[4], v[5], v[6], v[7]);
  }
}

__global__ void q80_dequant_tiled_kernel(const unsigned char* __restrict__ tiled, float* __restrict__ out, int out_dim,
                                         int in_dim, int nchunks) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)out_dim * in_dim) return;
  int row = (int)(i / in_dim), col = (int)(i - (size_t)row * in_dim);
  const int chunk = col >> 8;
  out[i] = tiled_weight<FMT_Q80>(tiled + ((size_t)(row >> 7) * nchunks + chunk) * Fmt<FMT_Q80>::kStageBytes, row & 127, col & 255);
}

// Q5_K super-blocks in the streaming layout {16-byte header, 8 x 16 bytes of nibbles, 8 x 4 bytes of
// fifth bits} -> stages; a thread per byte of nibbles (two elements), of bits (eight) and per header.
__global__ void q5k_tile_kernel(const unsigned char* __restrict__ blocks, unsigned char* __restrict__ tiled, int out_dim,
                                int ntiles, int nchunks) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kPer = 128 + 32 + 1;
  size_t nstages = (size_t)ntiles * nchunks;
  if (idx >= nstages * (128 * kPer)) return;
  size_t stg = idx / (128 * kPer);
  int rem = (int)(idx - stg * (128 * kPer));
  int tile = (int)(stg / nchunks), chunk = (int)(stg - (size_t)tile * nchunks);
  int r = rem / kPer, i = rem - r * kPer, row = tile * 128 + r;
  unsigned char* dst = tiled + stg * Fmt<FMT_Q5K>::kStageBytes;
  const unsigned char* src = blocks + ((size_t)row * nchunks + chunk) * 176;
  const bool in = row < out_dim;
  auto nib = [&](int k) { return (uint32_t)(src[16 + (k >> 1)] >> (4 * (k & 1))) & 0xFu; };
  auto fifth = [&](int k) { return (uint32_t)(src[144 + (k >> 3)] >> (k & 7)) & 1u; };
  if (i < 128) {
    const int k = (i >> 4) * 32 + (i & 15);  // and k + 16
    dst[kq_byte(r, k)] = in ? (unsigned char)(nib(k) | (nib(k + 16) << 4)) : 0;
  } else if (i < 160) {
    const int k = (i - 128) / 16 * 128 + (i & 15);  // of units 0 to 3 of the block, low and high
    uint32_t b = 0;
    for (int f = 0; f < 8 && in; ++f) b |= fifth(k + (f >> 1) * 32 + (f & 1) * 16) << f;
    dst[q5k_bit_byte(r, k)] = (unsigned char)b;
  } else {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (in) v = *reinterpret_cast<const uint4*>(src);
    *reinterpret_cast<uint4*>(dst + Fmt<FMT_Q5K>::kStageWBytes + r * 16) = v;
  }
}

// Q6_K planes (low nibbles, two-bit highs, int8 scales, f16 d) -> stages; a thread per byte of nibbles (two elements), of bits (four) and
// per row's scales.
__global__ void q6k_tile_kernel(const unsigned char* __restrict__ lo, const unsigned char* __restrict__ hi,
                                const signed char* __restrict__ sc, const uint16_t* __restrict__ dd,
                                unsigned char* __restrict__ tiled, int out_dim, int in_dim, int ntiles, int nchunks) {
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr int kPer = 128 + 64 + 1;
  size_t nstages = (size_t)ntiles * nchunks;
  if (idx >= nstages * (128 * kPer)) return;
  size_t stg = idx / (128 * kPer);
  int rem = (int)(idx - stg * (128 * kPer));
  int tile = (int)(stg / nchunks), chunk = (int)(stg - (size_t)tile * nchunks);
  int r = rem / kPer, i = rem - r * kPer, row = tile * 128 + r;
  unsigned char* dst = tiled + stg * Fmt<FMT_Q6K>::kStageBytes;
  const bool in = row < out_dim;
  const unsigned char *l = lo + (size_t)row * (in_dim / 2) + chunk * 128, *h = hi + (size_t)row * (in_dim / 4) + chunk * 64;
  auto nib = [&](int k) { return (uint32_t)(l[k >> 1] >> (4 * (k & 1))) & 0xFu; };
  auto two = [&](int k) { return (uint32_t)(h[k >> 2] >> (2 * (k & 3))) & 3u; };
  if (i < 128) {
    const int k = (i >> 4) * 32 + (i & 15);
    dst[kq_byte(r, k)] = in ? (unsigned char)(nib(k) | (nib(k + 16) << 4)) : 0;
  } else if (i < 192) {
    const int k = (i - 128) / 16 * 64 + (i & 15);
    uint32_t b = 0;
    for (int f = 0; f < 4 && in; ++f) b |= two(k + (f >> 1) * 32 + (f & 1) * 16) << (2 * f);
    dst[q6k_bits_byte(r, k)] = (unsigned char)b;
  } else {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (in) v = *reinterpret_cast<const uint4*>(sc + (size_t)row * (in_dim / 16) + chunk * 16);
    *reinterpret_cast<uint4*>(dst + Fmt<FMT_Q6K>::kStageWBytes + r * 16) = v;
    *reinterpret_cast<uint16_t*>(dst + Fmt<FMT_Q6K>::kDOff + r * 2) = in ? dd[(size_t)row * nchunks + chunk] : (uint16_t)0;
  }
}

// dequantRowQ5K / dequantRowQ6K from the tiled layouts (loader/gguf/quant_matrix.go:331-426), the
// roundings of the streaming layouts' kernels.
__global__ void q5k_dequant_tiled_kernel(const unsigned char* __restrict__ tiled, float* __restrict__ out, int out_dim,
                                         int in_dim, int nchunks) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)out_dim * in_dim) return;
  int row = (int)(i / in_dim), col = (int)(i - (size_t)row * in_dim);
  int chunk = col >> 8, k = col & 255, step = k >> 5, r = row & 127;
  const unsigned char* stg = tiled + ((size_t)(row >> 7) * nchunks + chunk) * Fmt<FMT_Q5K>::kStageBytes;
  const uint4 h = *reinterpret_cast<const uint4*>(stg + Fmt<FMT_Q5K>::kStageWBytes + r * 16);
  const int bit = 12 * step, wi = bit >> 5, sh = bit & 31;
  const uint32_t lo = wi == 0 ? h.y : wi == 1 ? h.z : h.w, hi = wi == 0 ? h.z : wi == 1 ? h.w : 0u;
  const uint32_t f = __funnelshift_r(lo, hi, sh) & 0xFFFu;
  const float sd = __fmul_rn((float)(f & 63u), __half2float(__ushort_as_half((unsigned short)(h.x & 0xFFFFu))));
  const float md = __fmul_rn((float)(f >> 6), __half2float(__ushort_as_half((unsigned short)(h.x >> 16))));
  const uint32_t q = ((stg[kq_byte(r, k)] >> (kq_upper(k) ? 4 : 0)) & 0xFu) | (((stg[q5k_bit_byte(r, k)] >> q5k_bit(k)) & 1u) << 4);
  out[i] = __fsub_rn(__fmul_rn(sd, (float)q), md);
}

__global__ void q6k_dequant_tiled_kernel(const unsigned char* __restrict__ tiled, float* __restrict__ out, int out_dim,
                                         int in_dim, int nchunks) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (size_t)out_dim * in_dim) return;
  int row = (int)(i / in_dim), col = (int)(i - (size_t)row * in_dim);
  const int chunk = col >> 8;
  out[i] = tiled_weight<FMT_Q6K>(tiled + ((size_t)(row >> 7) * nchunks + chunk) * Fmt<FMT_Q6K>::kStageBytes, row & 127, col & 255);
}

bool gguf_mma_supported(int qtype, int in_dim) {
  return (qtype == GOPH_GGUF_Q4_K || qtype == GOPH_GGUF_Q8_0 || qtype == GOPH_GGUF_Q5_K || qtype == GOPH_GGUF_Q6_K) &&
         (in_dim % kChunkK == 0 || (qtype == GOPH_GGUF_Q8_0 && in_dim % 32 == 0)) && in_dim <= kMaxPrepIn;
}

int gguf_mma_make_tiled(goph_gguf_matrix* m) {
  const int ntiles = (m->out_dim + kTileRows - 1) / kTileRows, nchunks = (m->in_dim + kChunkK - 1) / kChunkK;
  const bool q4 = m->qtype == GOPH_GGUF_Q4_K;
  const size_t stage = q4 ? Fmt<FMT_Q4K>::kStageBytes : m->qtype == GOPH_GGUF_Q5_K ? Fmt<FMT_Q5K>::kStageBytes : m->qtype == GOPH_GGUF_Q6_K ? Fmt<FMT_Q6K>::kStageBytes : Fmt<FMT_Q80>::kStageBytes;
  const size_t bytes = (size_t)ntiles * nchunks * stage;
  unsigned char* t = nullptr;
  GOPH_CUDA(cudaMalloc(&t, bytes));
  if (q4) {
    size_t threads = (size_t)ntiles * nchunks * 128 * 9;
    q4k_tile_kernel<<<(unsigned)((threads + 255) / 256), 256>>>(m->data, t, m->out_dim, ntiles, nchunks);
  } else if (m->qtype == GOPH_GGUF_Q5_K) {
    size_t threads = (size_t)ntiles * nchunks * 128 * 161;
    q5k_tile_kernel<<<(unsigned)((threads + 255) / 256), 256>>>(m->data, t, m->out_dim, ntiles, nchunks);
  } else if (m->qtype == GOPH_GGUF_Q6_K) {
    // planes behind one another: low nibbles in data; highs, int8 scales, f16 d in d16's buffer
    const size_t n = (size_t)m->out_dim * m->in_dim;
    const unsigned char* hi = reinterpret_cast<const unsigned char*>(m->d16);
    size_t threads = (size_t)ntiles * nchunks * 128 * 193;
    q6k_tile_kernel<<<(unsigned)((threads + 255) / 256), 256>>>(m->data, hi, reinterpret_cast<const signed char*>(hi + n / 4),
                                                                reinterpret_cast<const uint16_t*>(hi + n / 4 + n / 16), t, m->out_dim,
                                                                m->in_dim, ntiles, nchunks);
  } else {
    size_t threads = (size_t)ntiles * nchunks * 128 * 16;
    q80_tile_kernel<<<(unsigned)((threads + 255) / 256), 256>>>(m->data, m->d16, t, m->out_dim, m->in_dim, ntiles, nchunks);
  }
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaFree(t);
    return fail_cuda(e, "gguf tile kernel");
  }
  m->tiled = t;
  m->bytes = bytes;
  return GOPH_OK;
}

int gguf_mma_launch(const goph_gguf_matrix* m, float* out, const float* x, int batch, int digits, cudaStream_t stream,
                    SharedX* shared) {
  if (!m->tiled) return fail(GOPH_E_UNSUPPORTED, "matrix is not in the tiled layout");
  RowWeights d;
  d.device = m->device;
  d.in_dim = m->in_dim;
  d.n = 1;
  d.seg[0] = RowSeg{m->tiled, out, m->out_dim, 0};
  d.unordered = m->unordered;
  if (m->qtype == GOPH_GGUF_Q4_K) return rows_launch<FMT_Q4K, true>(d, x, batch, digits, stream, shared);
  if (m->qtype == GOPH_GGUF_Q5_K) return rows_launch<FMT_Q5K, true>(d, x, batch, digits, stream, shared);
  if (m->qtype == GOPH_GGUF_Q6_K) return rows_launch<FMT_Q6K, true>(d, x, batch, digits, stream, shared);
  return rows_launch<FMT_Q80, true>(d, x, batch, digits, stream, shared);
}

int gguf_mma_dequant(const goph_gguf_matrix* m, float* out, cudaStream_t stream) {
  const int nchunks = (m->in_dim + kChunkK - 1) / kChunkK;
  if (m->qtype == GOPH_GGUF_Q4_K) {
    size_t units = (size_t)m->out_dim * (m->in_dim / 32);
    q4k_dequant_tiled_kernel<<<(unsigned)((units + 255) / 256), 256, 0, stream>>>(m->tiled, out, m->out_dim, m->in_dim, nchunks);
  } else if (m->qtype == GOPH_GGUF_Q5_K || m->qtype == GOPH_GGUF_Q6_K) {
    size_t n = (size_t)m->out_dim * m->in_dim;
    if (m->qtype == GOPH_GGUF_Q5_K)
      q5k_dequant_tiled_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(m->tiled, out, m->out_dim, m->in_dim, nchunks);
    else
      q6k_dequant_tiled_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(m->tiled, out, m->out_dim, m->in_dim, nchunks);
  } else {
    size_t n = (size_t)m->out_dim * m->in_dim;
    q80_dequant_tiled_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(m->tiled, out, m->out_dim, m->in_dim, nchunks);
  }
  GOPH_CUDA(cudaGetLastError());
  return GOPH_OK;
}

// ---- grouped launches over a work list (GGUF experts stacked in one matrix) -------------------------------

// Measured with the products behind it (B200, 128 experts of 2048/768, Q4_K gate|up and Q8_0 down, us a call, CUDA-core kernels
// in front): 16 items 24.8 -> 17.5 and 21.9 -> 11.6, 64 items 76.5 -> 38.6 and 71 -> 20.4, 256 items 248 -> 82.7 and 257 -> 49.6.
// Bound by the weights of the distinct experts, whose tiles come once per entry, and the end of every item (900 cycles).
// A CTA per item of the list: the list is cut into entries of up to MB items of one expert, numbered by their first
// items, and the item's activations become digits, sums and scales of its entry.  Every CTA finds its own place in the
// list (up to kMaxWorkList words); the first also counts the entries.
template <int FMT, int MB>
__global__ void __launch_bounds__(256)
work_prep_kernel(const __grid_constant__ MmaWorkLaunch g, MmaWorkEntry* __restrict__ work, int* __restrict__ count, unsigned char* __restrict__ xb, size_t gxb,
                 unsigned long long stage_bytes) {
  __shared__ __align__(16) int ex[kMaxWorkList], rank[kMaxWorkList];
  __shared__ int s_leader;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, w = blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  for (int t = tid; t < kMaxWorkList; t += 256) {
    uint32_t e = 0xFFFFFFFFu;
    if (t < g.items) e = g.experts ? __ldg(g.experts + t) : 0u;
    ex[t] = e < (uint32_t)g.active ? (int)e : -1;
  }
  __syncthreads();
  for (int t = tid; t < g.items; t += 256) {  // an item's place among its expert's
    int r = 0;
    const int e = ex[t];
    for (int u = 0; u < t; u += 4) {
      const int4 q = *reinterpret_cast<const int4*>(ex + u);
      r += (q.x == e) + (u + 1 < t && q.y == e) + (u + 2 < t && q.z == e) + (u + 3 < t && q.w == e);
    }
    rank[t] = e < 0 ? -1 : r;
  }
  __syncthreads();
  const int e = ex[w], first = e < 0 ? 0 : rank[w] / MB * MB;
  int leaders = 0, id = 0, mine = 0;
  for (int t0 = 0; t0 < g.items; t0 += 256) {
    const int t = t0 + tid;
    const bool in = t < g.items && ex[t] >= 0, same = in && ex[t] == e && rank[t] >= first && rank[t] < first + MB;
    if (same && rank[t] == first) s_leader = t;
    leaders += __syncthreads_count(in && rank[t] % MB == 0);
    mine += __syncthreads_count(same);
  }
  if (w == 0 && tid == 0) *count = leaders;
  if (e < 0) {
    if (tid == 0) atomicCAS(g.status, 0, 601);
    return;
  }
  const int leader = s_leader, m = rank[w] - first;
  for (int t0 = 0; t0 < leader; t0 += 256) {
    const int t = t0 + tid;
    id += __syncthreads_count(t < leader && ex[t] >= 0 && rank[t] % MB == 0);
  }
  MmaWorkEntry* we = work + id;
  if (tid == 0) {
    if (m == 0) {
      for (int k = 0; k < 2; ++k) we->g.w[k] = g.tiled + ((size_t)e * g.mats + k) * (g.rows / kTileRows) * (g.in_dim / kChunkK) * stage_bytes;
      we->g.count = mine;
      we->g.expert = e;
    }
    we->g.item[m] = w;
    if (g.pos) {
      const unsigned long long at = (unsigned long long)__ldg(g.pos + w) * (unsigned long long)g.rows, left = at < g.dst_len ? g.dst_len - at : 0;
      if (left < (unsigned long long)g.rows) atomicCAS(g.status, 0, 602);
      we->dst[m] = g.out + (left ? at : 0);
      we->room[m] = left < (unsigned long long)g.rows ? (int)left : g.rows;
      we->weight[m] = __ldg(g.weight + w);
    }
  }
#pragma unroll 1
  for (int c = warp; c < g.in_dim / kChunkK; c += 8) {
    float v[8];
    load_eight(g.x + (size_t)w * g.in_dim + c * kChunkK + lane * 8, v);
    prep_chunk<FMT, MB>(v, lane, xb + (size_t)id * gxb + (size_t)c * XBlock<FMT, MB>::kBytes, m, 4);
  }
}

// A list's launches, and where their parts lie in the scratch: entries, their number, prepared activations.
struct WorkPlan {
  MmaArgs a;
  size_t smem, count_at, xb_at, bytes;
};
template <int FMT, int MB>
static WorkPlan plan_work(const MmaWorkLaunch& g) {
  typedef RowSmem<FMT, MB, false, true> M;
  WorkPlan p;
  memset(&p, 0, sizeof p);
  MmaArgs& a = p.a;
  a.nseg = 1;
  a.seg[0].out = g.out;
  a.seg[0].out_dim = g.rows;
  a.in_dim = g.in_dim;
  a.batch = MB;
  a.digits = 4;
  a.ntiles = a.gtpe = g.rows / kTileRows;
  a.nchunks = g.in_dim / kChunkK;
  a.splits = 1;
  a.gmats = g.mats;
  a.gdirect = g.pos ? 3 : 2;
  a.gxb = (size_t)a.nchunks * XBlock<FMT, MB>::kBytes;
  // at most so many entries: every expert may have one that is not full
  const int most_entries = (int)(((long long)g.items + (long long)(g.active < g.items ? g.active : g.items) * (MB - 1)) / MB);
  a.gmax = most_entries < g.items ? most_entries : g.items;
  a.items = a.gmax * g.mats * a.ntiles;
  a.stages = M::stages(kHalfSmem, 0, 0) >= 4 ? M::stages(kHalfSmem, 0, 0) : M::stages(kWholeSmem, 0, 0);
  p.smem = M::bytes(a.stages, 0, 0);
  auto place = [&](size_t bytes) {
    const size_t at = p.bytes;
    p.bytes += (bytes + 255) & ~(size_t)255;
    return at;
  };
  place((size_t)a.gmax * sizeof(MmaWorkEntry));
  p.count_at = place(sizeof(int));
  p.xb_at = place((size_t)a.gmax * a.gxb);
  return p;
}

template <int FMT, int MB>
static int launch_work(int device, const MmaWorkLaunch& g, unsigned char* scratch, int* status, cudaStream_t stream) {
  WorkPlan p = plan_work<FMT, MB>(g);
  MmaArgs& a = p.a;
  MmaWorkEntry* work = reinterpret_cast<MmaWorkEntry*>(scratch);
  int* count = reinterpret_cast<int*>(scratch + p.count_at);
  unsigned char* xb = scratch + p.xb_at;
  a.status = status;
  a.gwork = reinterpret_cast<const MmaGroupEntry*>(work);
  a.gcount = count;
  a.xb = xb;
  auto kern = mlx_mma_kernel<FMT, MB, false, true>;
  GOPH_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)p.smem));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(g.items);
  cfg.blockDim = dim3(256);
  note_launch();
  GOPH_CUDA(cudaLaunchKernelEx(&cfg, work_prep_kernel<FMT, MB>, g, work, count, xb, a.gxb, (unsigned long long)Fmt<FMT>::kStageBytes));
  const int slots = device_state(device).sm_count * (p.smem <= kHalfSmem ? 2 : 1), most = a.items / (g.pos ? 1 : 2);
  cfg.gridDim = dim3(most < slots ? most : slots);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = p.smem;
  note_launch();
  GOPH_CUDA(cudaLaunchKernelEx(&cfg, kern, a, NoMaps()));
  return GOPH_OK;
}

// Entries of two items; of four for Q8_0 (whose kernel spills 84 bytes a thread) where experts have three and more on average.  (Q4_K, whose scales want registers
// beside a chunk's own sums, spills more: entries of four and eight items were 7 to 30 % slower, as were those of eight for Q8_0.)
static bool wide_entries(const MmaWorkLaunch& g) { return g.items >= 3 * g.active; }

size_t gguf_mma_work_bytes(const goph_gguf_matrix* m, const MmaWorkLaunch& g) {
  if (!m->tiled || (m->qtype != GOPH_GGUF_Q4_K && m->qtype != GOPH_GGUF_Q8_0) || g.items > kMaxWorkList || g.rows % kTileRows || g.in_dim % kChunkK ||
      g.in_dim > 16384)
    return 0;
  // A short list leaves most SMs idle at a tile (with gate and up: a pair of tiles) a CTA, or is over before the two launches
  // are.  The CUDA-core kernels spread a warp to a row and read an expert's rows once for four of its items, so that few
  // experts with several items each suit them longer; Q4_K's walk 1024 elements at a time and waste the rest of the last.  4552 lists of 1 to
  // 64 items, 1 to 128 experts, 256 to 12288 rows and 512 to 4096 elements were measured, 3203 lie past these lines and none of them is slower for it.  B200, us,
  // CUDA cores / these.  Two items an expert and more: gate|up Q4_K 2 experts, 8 items of 1024x2048 12.4 / 17.3; Q8_0 2, 16 of 1024x512 10.4 / 12.0; scatter
  // Q4_K 8, 32 of 512x1024 8.3 / 10.6.  More items than experts: gate|up Q4_K 8, 12 of 1024x1024 12.4 / 12.8; Q8_0 scatter 4, 6 of 1536x1024 8.3 / 9.5.  Fewer: gate|up Q4_K
  // 8, 6 of 1536x2048 14.4 / 17.5, 32, 2 of 3072x2048 16.5 / 16.9, 128, 16 of 768x2048 26.3 / 17.2, 128, 8 of 768x2560 23.4 / 19.8; scatter Q4_K 32, 16 of
  // 512x1024 9.0 / 10.2, Q8_0 32, 5 of 2048x768 12.4 / 9.0.
  const bool q4 = m->qtype == GOPH_GGUF_Q4_K, scatter = g.pos != nullptr;
  const long tiles = (long)g.items * (g.rows / kTileRows), size = (long)g.items * g.rows * g.in_dim;
  int least_tiles, least_mi;
  if (g.items >= 2l * g.active) {
    least_tiles = 144;
    least_mi = 10;
  } else if (g.items > g.active) {
    least_tiles = q4 ? 96 : 64;
    least_mi = q4 ? 8 : 10;
  } else {
    least_tiles = !q4 || g.in_dim % 1024 ? (scatter ? 64 : 48) : 4l * g.items > g.active ? 80 : scatter ? 72 : 56;
    least_mi = scatter ? 6 : 8;
  }
  if (tiles < least_tiles || size < (long)least_mi << 20) return 0;
  if (m->qtype == GOPH_GGUF_Q4_K) return plan_work<FMT_Q4K, 2>(g).bytes;
  return wide_entries(g) ? plan_work<FMT_Q80, 4>(g).bytes : plan_work<FMT_Q80, 2>(g).bytes;
}

int gguf_mma_launch_work(const goph_gguf_matrix* m, const MmaWorkLaunch& g0, unsigned char* scratch, int* status, cudaStream_t stream) {
  MmaWorkLaunch g = g0;
  g.tiled = m->tiled;
  if (m->qtype == GOPH_GGUF_Q4_K) return launch_work<FMT_Q4K, 2>(m->device, g, scratch, status, stream);
  return wide_entries(g) ? launch_work<FMT_Q80, 4>(m->device, g, scratch, status, stream) : launch_work<FMT_Q80, 2>(m->device, g, scratch, status, stream);
}

// ---- GEMV without any allocation ---------------------------------------------------------------
// Some callers must not allocate device memory when they run a product: a serving loop that has
// handed the whole memory budget to its KV and expert pools (an allocation could fail, or block
// behind a free), a thread that may not take the allocator's device-wide synchronisation in the
// middle of a decode step, or code that has begun capturing a stream.  For them the scratch of the
// tensor-core GEMV (status word, tile counters, the prepared activation digits and tables, the
// split-K partial sums) lives in this file-scope device array instead of in buffers obtained with
// cudaMalloc.  Every GPU that loads the library carries the array until the process exits.
constexpr int kNoAllocMaxIn = 16384;     // largest in_dim the entry point accepts
constexpr int kNoAllocMaxTiles = 4096;   // largest ceil(out_dim / 128)
constexpr int kNoAllocMaxItems = 320;    // (tile, split) items that may have partial sums at once
constexpr size_t kNaStatusOff = 0;
constexpr size_t kNaCountersOff = 256;
constexpr size_t kNaXbOff = kNaCountersOff + (size_t)kNoAllocMaxItems * kConsumers * 4;  // (tiles that are cut are fewer than the items)
constexpr size_t kNaPartOff = kNaXbOff + (size_t)(kNoAllocMaxIn / kChunkK) * XBlock<FMT_MLX4, 1>::kBytes;
constexpr size_t kNoAllocBytes = kNaPartOff + (size_t)kNoAllocMaxItems * RowCfg<FMT_MLX4, 1, false>::kRecv;
static_assert(kNaXbOff % 256 == 0 && kNaPartOff % 256 == 0, "256-byte aligned regions");
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Device address of the array on `device` (which must be current).  In host code the array's
// name is only a handle for the runtime, never a pointer a kernel could use, so the address is
// looked up once per device with cudaGetSymbolAddress and cached.
static int noalloc_base(int device, unsigned char** base) {
  static unsigned char* cached[kMaxDevices] = {};
  if (!cached[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return fail_cuda(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
    if (!p) return fail(GOPH_E_CUDA, "cudaGetSymbolAddress returned a null address for the scratch array");
    cached[device] = static_cast<unsigned char*>(p);
  }
  *base = cached[device];
  return GOPH_OK;
}

static int launch_noalloc(const goph_mlx_weight* w, float* out, const float* x, unsigned char* base, int digits, cudaStream_t stream) {
  MmaArgs a;
  memset(&a, 0, sizeof a);
  a.x = x;
  a.status = reinterpret_cast<int*>(base + kNaStatusOff);
  a.counters = reinterpret_cast<unsigned int*>(base + kNaCountersOff);
  a.xb = base + kNaXbOff;
  a.scratch = reinterpret_cast<float*>(base + kNaPartOff);
  a.batch = 1;
  a.digits = digits == 3 ? 3 : 4;
  // The array keeps whatever the last call left: the arrival counters have to start at zero (the prepared activations and
  // partial sums are fully rewritten before they are read).  The status word is
  // left alone: it is zero when the library is loaded and sticky once a wait has given up, like the
  // allocated path's; goph_mlx_gemv_noalloc_status reads it.
  GOPH_CUDA(cudaMemsetAsync(base + kNaCountersOff, 0, kNaXbOff - kNaCountersOff, stream));
  RowWeights d;
  d.device = w->device;
  d.in_dim = w->in_dim;
  d.n = 1;
  d.seg[0] = RowSeg{w->tiled, out, w->out_dim, 0};
  d.scratch_bytes = kNoAllocBytes - kNaPartOff;
  d.counters = kNoAllocMaxItems * kConsumers;
  SharedX xs;
  xs.written = floats_meet(out, w->out_dim, x, w->in_dim);
  return rows_slice<FMT_MLX4, true>(d, a, stream, &xs);
}

}  // namespace goph

using namespace goph;

GOPH_API int goph_mlx_gemv_noalloc_status(int device, int* out_status) {
  clear_error();
  if (!out_status) return fail(GOPH_E_INVALID, "goph_mlx_gemv_noalloc_status: nil result pointer");
  if (int rc = use_device(device)) return rc;
  unsigned char* base = nullptr;
  if (int rc = noalloc_base(device, &base)) return rc;
  GOPH_CUDA(cudaMemcpy(out_status, base + kNaStatusOff, sizeof(int), cudaMemcpyDeviceToHost));
  return GOPH_OK;
}

GOPH_API int goph_mlx_gemv_noalloc(float* out_dev, uint64_t out_len, const float* x_dev, uint64_t x_len,
                                   const goph_mlx_weight* w, void* stream) {
  clear_error();
  if (!w || w->magic != kMagicMLX) return fail(GOPH_E_INVALID, "invalid MLX weight handle");
  if (!w->tiled)
    return fail(GOPH_E_UNSUPPORTED,
                "goph_mlx_gemv_noalloc needs a weight in the tiled layout (group size 64, in_dim a multiple of 256, "
                "uploaded with mlx_layout 0 or 2); this one is row-major");
  if (w->in_dim > kNoAllocMaxIn)
    return fail(GOPH_E_UNSUPPORTED, "goph_mlx_gemv_noalloc: in_dim=%d is above the built-in scratch limit of %d", w->in_dim,
                kNoAllocMaxIn);
  if ((w->out_dim + kTileRows - 1) / kTileRows > kNoAllocMaxTiles)
    return fail(GOPH_E_UNSUPPORTED, "goph_mlx_gemv_noalloc: out_dim=%d is above the built-in scratch limit of %d", w->out_dim,
                kNoAllocMaxTiles * kTileRows);
  if (!x_dev || x_len < (uint64_t)w->in_dim || !out_dev || out_len < (uint64_t)w->out_dim)
    return fail(GOPH_E_INVALID, "buffers x=%llu/%d out=%llu/%d", (unsigned long long)x_len, w->in_dim,
                (unsigned long long)out_len, w->out_dim);
  if ((uintptr_t)x_dev % 16) return fail(GOPH_E_INVALID, "goph_mlx_gemv_noalloc: x must be 16-byte aligned");
  if (int rc = use_device(w->device)) return rc;
  unsigned char* base = nullptr;
  if (int rc = noalloc_base(w->device, &base)) return rc;
  return launch_noalloc(w, out_dev, x_dev, base, options().mlx_digits, (cudaStream_t)stream);
}
