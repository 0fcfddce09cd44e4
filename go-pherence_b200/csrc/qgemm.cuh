// Quantised weights times several activation rows (prefill chunks, verifier batches) on the tensor
// cores, for every weight format and both device layouts; implemented in qgemm.cu.
#pragma once

#include <mutex>

#include "goph_internal.cuh"

namespace goph {

// Q_MLX4F: MLX 4-bit weights whose scales are zero or of magnitude 2^-27 to 7.875 (goph_mlx_weight::foldable)
enum QFormat { Q_MLX4 = 0, Q_Q4K = 1, Q_Q5K = 2, Q_Q6K = 3, Q_Q80 = 4, Q_FP8 = 5, Q_MLX4F = 6 };

// A weight matrix as the kernel sees it.  maps: of the other layouts, made at upload.  tiled: `w` is the format's tiled layout; else `w` and `aux`
// are the row-major / streaming layout's buffers (MLX: words and the bf16 {scale,bias} table; Q4_K,
// Q5_K: blocks; Q6_K: low nibbles, and the highs, scales and d one plane after another; Q8_0: biased
// bytes and f16 scales; FP8: bytes).
struct QWeight {
  int fmt;
  bool tiled;
  const void* w;
  const void* aux;
  const float* scale;  // FP8: [out_dim]
  const float* bias;   // FP8: [out_dim] or nullptr
  int device, out_dim, in_dim;
  const QMaps* maps;
  bool unordered = false;  // tiled: the scratch is the stream's all the same
};

// The tensor maps of a weight in its row-major or streaming layout (w and aux as in QWeight).  maps->ok is false where there
// are none (no such driver call, rows that are no whole 16-byte units): such a weight is not for this kernel.
// MLX: aux has rows of whole 16-byte units (in_dim / 64 entries, rounded up to four).
void qgemm_maps(int fmt, const void* w, const void* aux, int out_dim, int in_dim, QMaps* maps);

// Whether `batch` activation rows of such a weight go to this kernel; the others are the business of the kernels
// for few rows (integer tensor-core GEMV, CUDA-core streaming, FP8 pieces).  `weights` of one call that share x and could
// share a launch there count together, out_dim being the sum of theirs.
bool qgemm_wants(int fmt, bool tiled, bool x_bf16, long out_dim, int in_dim, int batch, int weights = 1);

// Layouts other than the tiled ones, and small tiled matrices: the scratch of a call on this stream (see the definition), which qgemm wants; if
// there is none, the call is the business of the kernels for few rows, which need none.
struct QBufs;
QBufs* qgemm_scratch(int device, cudaStream_t stream);

// The area itself, for other launches that prepare activations; enqueue is to be held from the first of them to the last.
constexpr size_t kStreamXbBytes = (size_t)24 << 20;  // of a stream's area
struct QScratch {
  unsigned char* bytes;  // kStreamXbBytes of them
  int* status;           // the area's status word, which qgemm_status reads
  std::mutex* enqueue;
};
QScratch qgemm_scratch_area(QBufs* b);

// A weight handle of any format was made (+1) or is being freed (-1).
void qgemm_weights(int device, int change);

// out[i] [batch][out_dim] = x [batch][in_dim] . W[i]^T for n weights of one device and in_dim, x f32 or bf16 bit
// patterns, 16-byte aligned, prepared once for weights of the same format and kind of layout.  rows: qgemm_scratch's
// answer where a weight is not tiled or is unordered.
int qgemm(int n, const QWeight* w, float* const* out, const void* x, bool x_bf16, int batch, QBufs* rows, cudaStream_t stream);

int qgemm_status(int device);
void qgemm_status_clear(int device);

}  // namespace goph
