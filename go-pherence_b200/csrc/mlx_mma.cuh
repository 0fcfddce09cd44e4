// Tensor-core products of few activation rows (MLX, GGUF, FP8); implemented in mlx_mma.cu.
#pragma once

#include "goph_internal.cuh"

namespace goph {

// True when the weight's shape allows the tiled layout of the tensor-core kernel (bf16
// scale/bias table, group size 64, in_dim a multiple of 256).
bool mlx_mma_supported(const goph_mlx_weight* w);
// Builds the tiled copy from the row-major buffers of w (which the caller then frees).
int mlx_mma_make_tiled(goph_mlx_weight* w);
// Byte offsets inside the tiled layout (shared with the dequantisation kernel).
constexpr int kMlxTileRows = 128, kMlxChunkK = 256, kMlxBlockW = 128 * 128, kMlxBlockBytes = 128 * 128 + 128 * 16;
__host__ __device__ inline size_t mlx_tiled_word_offset(int row, int col, int nchunks) {
  size_t blk = (size_t)(row >> 7) * nchunks + (col >> 8);
  int r = row & 127, u = (col & 255) >> 5, w = (col & 31) >> 3;
  return blk * kMlxBlockBytes + r * 128 + ((u ^ (r & 7)) << 4) + w * 4;
}
__host__ __device__ inline size_t mlx_tiled_meta_offset(int row, int col, int nchunks) {
  size_t blk = (size_t)(row >> 7) * nchunks + (col >> 8);
  return blk * kMlxBlockBytes + kMlxBlockW + (row & 127) * 16 + ((col & 255) >> 6) * 4;
}
// What the launches of one call know of the x they share (same batch, same in_dim, same kind of weight).
struct SharedX {
  bool prepared = false;  // a launch in front on this stream has left it prepared in the device's scratch (one that prepares its own K ranges leaves nothing there)
  bool written = false;   // an output of the call overlaps it: no product may read it, it is prepared before the first of them
};
// out[batch][out_dim] = x[batch][in_dim] * W^T.  digits: base-128 digits each activation is
// written in (4 = 27 bits under the group maximum, 3 = 20 bits).  shared: nullptr for a call of one weight.
int mlx_mma_launch(const goph_mlx_weight* w, float* out, const float* x, int batch, int digits, cudaStream_t stream,
                   SharedX* shared = nullptr);

// The same for n row-major weights of one device and in_dim that share x, in one launch for up to four of them: groups of 64, bf16 tables, tensor maps
// (mlx_mma_rows_ok).  No scratch: callers need no order between such calls.
inline bool mlx_mma_rows_ok(const goph_mlx_weight* w) { return !w->tiled && w->group_size == 64 && w->sb_bf16 && w->qmaps.ok && w->in_dim <= 65536; }
int mlx_mma_launch_rows(int n, const goph_mlx_weight* const* ws, float* const* outs, const float* x, int batch, int digits, cudaStream_t stream);
// FP8 linears of either layout (row-major: with tensor maps), f32 activations; row-major: no scratch.
int fp8_mma_launch_rows(const goph_fp8_linear* w, float* out, const float* x, int batch, cudaStream_t stream);
// Allocates the device's scratch (uploads do, so that no product of a weight that may be used under capture has to).
bool mlx_mma_ready(int device);

// ---- grouped launches: the selected experts of a mixture-of-experts layer --------------------
// One work entry = one expert (tiled matrices of equal shapes) and up to `rows` (2 or 4, the same
// for every entry of a call) of the (token, slot) items that chose it; an expert chosen by more
// items has several entries.
constexpr int kMoeMmaRowsMin = 2, kMoeMmaRowsMax = 4;
struct __align__(16) MmaGroupEntry {
  const unsigned char* w[3];  // tiled gate, up, down
  int count;                  // items of this entry, 1..rows
  int expert;
  int item[8];                // token * top_k + slot
};
// True when experts of [inter x hidden] / [hidden x inter] can run as grouped launches.
bool mlx_mma_grouped_supported(int hidden, int inter);
// Bytes of prepared activations one entry of `rows` items needs for an input of in_dim.
size_t mlx_mma_grouped_xb_bytes(int in_dim, int rows);
struct MmaGroupLaunch {
  const MmaGroupEntry* work;  // device
  const int* count;           // device: live entries
  int max_entries;            // entries the launch is sized for
  int entry_rows;             // items per entry: 2 or 4
  int first, mats;            // matrices of an entry this launch multiplies: w[first .. first + mats)
  int rows, in_dim;           // shape of each of them
  int phase;                  // 0: activations = row item / top_k of src; 1: silu(g) * u of src's row entry * entry_rows + m
  int top_k;
  const float* src;
  unsigned char* xb;          // [max_entries][xb_bytes]
  float* out;                 // phase 0: [max_entries * entry_rows][mats * rows]; phase 1: [items][rows]
};
// Two launches: the entries' activations as digits, sums and scales; then the products.
int mlx_mma_launch_grouped(int device, const MmaGroupLaunch& g, cudaStream_t stream);

// ---- grouped launches over a work list: GGUF experts stacked in one tiled matrix -------------------------
constexpr int kMaxWorkList = 512;
// Up to four items of one expert (g.w: its gate and up, or its matrix).
struct __align__(16) MmaWorkEntry {
  MmaGroupEntry g;    // item: place in the list
  float* dst[4];      // scatter: destination row of each item, how many of its elements there are, its weight
  int room[4];
  float weight[4];
};
struct MmaWorkLaunch {
  const unsigned char* tiled;  // (filled in)
  const float* x;              // [items][in_dim]
  const uint32_t* experts;     // [items], or nullptr: all 0
  const uint32_t* pos;         // scatter: destination row of each item; nullptr: out[items][rows] = gelu(gate) * up
  const float* weight;
  float* out;
  unsigned long long dst_len;
  int* status;                 // 601: expert outside the matrix, 602: destination outside out (skipped)
  int items, active, mats, rows, in_dim;  // experts, matrices of each (gate and up: 2), rows of each of them
};
// Scratch that gguf_mma_launch_work wants for this list; 0: it is a list for other kernels.
size_t gguf_mma_work_bytes(const goph_gguf_matrix* m, const MmaWorkLaunch& g);
// Two launches (entries and activations; products) with the caller's scratch, which is in use until they are through.
// status: the word a wait that gives up leaves its code in.
int gguf_mma_launch_work(const goph_gguf_matrix* m, const MmaWorkLaunch& g, unsigned char* scratch, int* status, cudaStream_t stream);

// Reads the device status word (0 = every wait completed); synchronises the copy stream.
int mlx_mma_status(int device);
void mlx_mma_status_clear(int device);

// GGUF matrices on the same kernel.  make_tiled builds m->tiled from the matrix's device
// buffers (which the caller then frees); dequant reproduces dequantRowQ4KTo / dequantRowQ8_0To.
bool gguf_mma_supported(int qtype, int in_dim);
int gguf_mma_make_tiled(goph_gguf_matrix* m);
int gguf_mma_launch(const goph_gguf_matrix* m, float* out, const float* x, int batch, int digits, cudaStream_t stream,
                    SharedX* shared = nullptr);
int gguf_mma_dequant(const goph_gguf_matrix* m, float* out, cudaStream_t stream);

}  // namespace goph
