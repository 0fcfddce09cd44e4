// Streaming GEMV / small-batch skeleton shared by the GGUF and FP8 formats.
//
// Same shape as the MLX kernel: a warp owns R rows at a time; lane l of iteration `it`
// owns one 16-byte unit (unit = 32*it + l) of each of those rows, so a warp instruction is
// a 512-byte coalesced, L1-bypassing load per row.  x is staged once per CTA in shared
// memory as f32 in the order [batch][it][slot][lane] (conflict-free LDS.128), with one
// float2 of per-unit constants beside it when the format needs them (offset removal and
// the affine term).  The next step's weights are in flight while the current step computes.
// The first step's weights are asked for before the kernel in front has ended (programmatic dependent launch; the
// kernel itself lets the next one start when it ends: asked for earlier, the next one's CTAs crowd onto a few SMs,
// Q8_0 1536x4096 12.4 us a call instead of 5.8).  Small matrices come here, so a call's own cost bounds most of
// them: two driver queries per launch, x read in 16-byte pieces 128 bytes apart.  Without these and with the early start
// (B200, us a call): Q4_K 2048x2048 6.2 -> 4.2, Q6_K 2048x2048 x2 8.2 -> 4.6, Q8_0 1536x4096 8.3 -> 5.8, Q5_K 1024x2816
// x8 16.4 -> 10.7, Q8_0 4096x1536 x3 10.3 -> 8.7.
//
// A format policy F provides:
//   kSlots                 float4 of x per unit (unit elements / 4)
//   kHasConsts             whether per-unit constants are needed
//   struct Row             per-row data of one unit (the 16 weight bytes + metadata)
//   load(a,row,unit,Row&)  issue the loads of one unit of one row
//   consts(se,so)          float2 from the even/odd-position sums of the unit's x
//   dot(Row, xs, c, acc)   acc[m] += contribution of this unit, for m < M
//   finish(a,row,v)        per-row epilogue (row scale, bias)
#pragma once

#include <string.h>

#include <mutex>

#include "goph_internal.cuh"

namespace goph {

constexpr int kGWarps = 8;
constexpr int kGThreads = kGWarps * 32;

struct StreamArgs {
  const uint8_t* w;     // weight bytes
  const void* aux;      // format metadata (Q8_0: f16 scales; FP8: f32 row scales)
  const float* bias;    // FP8 bias or nullptr
  float* out;           // [batch][rows]
  const float* x;       // [batch][in_dim]
  int rows, in_dim, batch;
  int units;            // 16-byte units per row
  int iters;            // ceil(units / 32)
  int x_aligned;
  int row_bytes;

};

template <class F>
__host__ __device__ inline size_t stream_smem_bytes(int M, int iters) {
  return (size_t)M * iters * (F::kSlots * 32 * 16 + (F::kHasConsts ? 32 * 8 : 0));
}

template <class F, int R, int M>
__global__ void __launch_bounds__(kGThreads)
stream_gemv_kernel(const __grid_constant__ StreamArgs a) {
  constexpr int S = F::kSlots;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* xs = reinterpret_cast<float4*>(smem_raw);
  float2* xc = reinterpret_cast<float2*>(smem_raw + (size_t)M * a.iters * S * 32 * 16);

  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // (uniform, for the compiler)
  const int iters = a.iters;
  const int tasks = (a.rows + R - 1) / R;
  const int task_stride = gridDim.x * kGWarps;
  int task = blockIdx.x * kGWarps + warp, it = 0;

  typename F::Row cur[R], nxt[R];
  auto load_tile = [&](int t, int i, typename F::Row (&dst)[R]) {
    int unit = i * 32 + lane;
    if (unit >= a.units) unit = a.units - 1;  // x is zero there
#pragma unroll
    for (int r = 0; r < R; ++r) {
      int row = t * R + r;
      if (row >= a.rows) row = a.rows - 1;
      F::load(a, row, unit, dst[r]);
    }
  };
  const bool has_work = task < tasks;
  if (has_work) load_tile(task, 0, cur);

  // ---- stage x (which the kernel in front may write): coalesced reads, kV of them in flight ----
  asm volatile("griddepcontrol.wait;" ::: "memory");
  {
    constexpr int kV = 4;
    const int per_m = iters * S * 32;  // float4s of a row, as float4 q of the row: slot q % S of unit q / S
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
#pragma unroll 1
      for (int q0 = threadIdx.x; q0 < per_m; q0 += kV * kGThreads) {
        float4 v[kV];
#pragma unroll
        for (int k = 0; k < kV; ++k) {
          const int q = q0 + k * kGThreads, unit = q / S;
          v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (m < a.batch && unit < a.units) {
            const float* p = a.x + (size_t)m * a.in_dim + (size_t)q * 4;
            v[k] = a.x_aligned ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
          }
        }
#pragma unroll
        for (int k = 0; k < kV; ++k) {
          const int q = q0 + k * kGThreads, unit = q / S;
          if (q < per_m) xs[(size_t)m * per_m + ((unit >> 5) * S + q % S) * 32 + (unit & 31)] = v[k];
        }
      }
    }
    __syncthreads();
    if (F::kHasConsts) {
      const int nsum = M * iters * 32;
      for (int idx = threadIdx.x; idx < nsum; idx += kGThreads) {
        int mi = idx >> 5, l = idx & 31;
        float se = 0.f, so = 0.f;
#pragma unroll
        for (int s = 0; s < S; ++s) {
          float4 v = xs[(mi * S + s) * 32 + l];
          se += v.x + v.z;
          so += v.y + v.w;
        }
        xc[idx] = F::consts(se, so);
      }
      __syncthreads();
    }
  }
  if (!has_work) return;

  float acc[R][M];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int m = 0; m < M; ++m) acc[r][m] = 0.f;

  while (true) {
    int ntask = task, nit = it + 1;
    if (nit == iters) {
      nit = 0;
      ntask = task + task_stride;
    }
    const bool more = ntask < tasks;
    if (more) load_tile(ntask, nit, nxt);

    float4 xv[M][S];
    float2 c[M];
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
      for (int s = 0; s < S; ++s) xv[m][s] = xs[((size_t)(m * iters + it) * S + s) * 32 + lane];
      c[m] = F::kHasConsts ? xc[(m * iters + it) * 32 + lane] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) F::template dot<M>(cur[r], xv, c, acc[r]);

    if (it == iters - 1) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        int row = task * R + r;
#pragma unroll
        for (int m = 0; m < M; ++m) {
          float v = warp_sum(acc[r][m]);
          acc[r][m] = 0.f;
          if (lane == 0 && row < a.rows && m < a.batch) a.out[(size_t)m * a.rows + row] = F::finish(a, row, v);
        }
      }
    }
    if (!more) break;
#pragma unroll
    for (int r = 0; r < R; ++r) cur[r] = nxt[r];
    task = ntask;
    it = nit;
  }
}

typedef void (*StreamKernel)(const StreamArgs);

template <class F>
static StreamKernel stream_pick(int R, int M) {
  switch (M) {
    case 1:
      return R == 4 ? (StreamKernel)stream_gemv_kernel<F, 4, 1> : R == 2 ? (StreamKernel)stream_gemv_kernel<F, 2, 1>
                                                                         : (StreamKernel)stream_gemv_kernel<F, 1, 1>;
    case 2:
      return R == 4 ? (StreamKernel)stream_gemv_kernel<F, 4, 2> : R == 2 ? (StreamKernel)stream_gemv_kernel<F, 2, 2>
                                                                         : (StreamKernel)stream_gemv_kernel<F, 1, 2>;
    case 4:
      return R >= 2 ? (StreamKernel)stream_gemv_kernel<F, 2, 4> : (StreamKernel)stream_gemv_kernel<F, 1, 4>;
    default:
      return R >= 2 ? (StreamKernel)stream_gemv_kernel<F, 2, 8> : (StreamKernel)stream_gemv_kernel<F, 1, 8>;
  }
}

// CTAs of kernel <F, R, M> an SM holds with `smem` bytes each.  The shared-memory limit of a kernel and the answer for
// the last size asked for are kept: the two driver calls cost more than the launch.
template <class F>
static int stream_occupancy(StreamKernel k, int R, int M, size_t smem, int device) {
  struct Known {
    size_t limit, smem;
    int per_sm;
  };
  static std::mutex mu;
  static Known known[kMaxDevices][3][4] = {};
  std::lock_guard<std::mutex> lock(mu);
  Known& e = known[device][R >> 1][M == 1 ? 0 : M == 2 ? 1 : M == 4 ? 2 : 3];
  if (e.limit < smem) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    e.limit = smem;
  }
  if (e.smem != smem) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kGThreads, smem) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    e.smem = smem;
    e.per_sm = n;
  }
  return e.per_sm;
}

// Runs x [batch,in] through the streaming kernel in batch tiles that fit shared memory.
// Returns GOPH_E_UNSUPPORTED when even one activation row does not fit.
template <class F>
static int stream_launch(StreamArgs a, int device, int batch, cudaStream_t stream, int force_rows = 0) {
  DeviceState& st = device_state(device);
  a.iters = (a.units + 31) / 32;
  if (stream_smem_bytes<F>(1, a.iters) > (size_t)kSmemBudget)
    return fail(GOPH_E_UNSUPPORTED, "in_dim=%d: one activation row does not fit in shared memory", a.in_dim);
  int tile = 8;
  while (tile > 1 && stream_smem_bytes<F>(tile, a.iters) > (size_t)kSmemBudget) tile >>= 1;
  const float* x0 = a.x;
  float* out0 = a.out;
  for (int b0 = 0; b0 < batch; b0 += tile) {
    int nb = batch - b0 < tile ? batch - b0 : tile;
    int M = nb <= 1 ? 1 : nb <= 2 ? 2 : nb <= 4 ? 4 : 8;
    int R = force_rows;
    if (R != 1 && R != 2 && R != 4) {
      long want = (long)st.sm_count * 2 * kGWarps * 2;
      R = a.rows / 4 >= want ? 4 : a.rows / 2 >= want ? 2 : 1;
    }
    if (M >= 4 && R == 4) R = 2;
    a.x = x0 + (size_t)b0 * a.in_dim;
    a.out = out0 + (size_t)b0 * a.rows;
    a.batch = nb;
    a.x_aligned = ((uintptr_t)a.x % 16) == 0;
    StreamKernel k = stream_pick<F>(R, M);
    size_t smem = stream_smem_bytes<F>(M, a.iters);
    const int per_sm = stream_occupancy<F>(k, R, M, smem, device);
    if (per_sm < 1) return fail(GOPH_E_UNSUPPORTED, "streaming kernel does not fit (smem %zu)", smem);
    int tasks = (a.rows + R - 1) / R;
    int grid = (tasks + kGWarps - 1) / kGWarps;
    if (grid > st.sm_count * per_sm) grid = st.sm_count * per_sm;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = options().pdl ? 1 : 0;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kGThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    note_launch();
    GOPH_CUDA(cudaLaunchKernelEx(&cfg, k, a));
  }
  return GOPH_OK;
}

}  // namespace goph
