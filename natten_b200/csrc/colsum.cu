// Column sums of a row-major [rows, cols] matrix of 16-bit floats, fp32 accumulation: the bias
// gradient of the layers' linear projections. HBM-bound, one read of the matrix.
//
// A block covers 256 columns (32 lanes of 16 bytes, 8 warps on 8 consecutive rows) of one slice of
// the rows; slices are cut so that about four blocks per SM are in flight, and their partial sums
// (fp32, [slices, cols]) are added in slice order by a second small kernel: the same bits every time,
// no atomics. A generic reduction over the slow axis of [100352, 384] takes 95 us (0.8 TB/s); this
// one reads the 77 MB at the copy rate.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace b200na {
namespace {

constexpr int kWarps = 8;
constexpr int kBlockCols = 256;   // 32 lanes x 8 elements
constexpr int kUnroll = 4;        // rows in flight per warp

struct Split {
  int slices;
  int64_t rows_per;   // rows of a slice, a multiple of kWarps
};
Split split_rows(int64_t rows, int cols) {
  const int64_t col_blocks = (cols + kBlockCols - 1) / kBlockCols;
  int64_t want = 592 / col_blocks;    // four blocks for each of 148 SMs
  const int64_t most = (rows + kWarps * kUnroll - 1) / (kWarps * kUnroll);
  if (want > most) want = most;
  if (want < 1) want = 1;
  Split s;
  s.rows_per = ((rows + want - 1) / want + kWarps - 1) / kWarps * kWarps;
  s.slices = (int)((rows + s.rows_per - 1) / s.rows_per);
  if (s.slices < 1) s.slices = 1;
  return s;
}

template <class T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <class T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

template <class T>
__global__ void __launch_bounds__(kWarps * 32) partial_kernel(const T* __restrict__ in,
                                                              float* __restrict__ part, int64_t rows,
                                                              int cols, int64_t rows_per) {
  __shared__ float sums[kWarps][kBlockCols];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col = blockIdx.x * kBlockCols + lane * 8;
  const int64_t first = blockIdx.y * rows_per;
  const int64_t last = first + rows_per < rows ? first + rows_per : rows;
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
  if (col < cols) {
    const T* p = in + col;
    int64_t r = first + warp;
    for (; r + (kUnroll - 1) * kWarps < last; r += kUnroll * kWarps) {
      uint4 x[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        x[u] = *reinterpret_cast<const uint4*>(p + (r + u * kWarps) * cols);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const T* v = reinterpret_cast<const T*>(&x[u]);
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[e] += to_f(v[e]);
      }
    }
    for (; r < last; r += kWarps) {
      const uint4 x = *reinterpret_cast<const uint4*>(p + r * cols);
      const T* v = reinterpret_cast<const T*>(&x);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += to_f(v[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) sums[warp][lane * 8 + e] = acc[e];
  __syncthreads();
  const int c = blockIdx.x * kBlockCols + threadIdx.x;
  if (c < cols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s += sums[w][threadIdx.x];
    part[(int64_t)blockIdx.y * cols + c] = s;
  }
}

// 32 columns per block, 32 warps over the slices, eight loads of a warp in flight. Latency is all there
// is here (0.9 MB from L2): with 8 warps and one running sum each, 592 slices of 128 columns took 11 us,
// more than the 26 MB that they are the sums of.
constexpr int kFinishWarps = 32, kFinishUnroll = 8;
template <class T>
__global__ void __launch_bounds__(kFinishWarps * 32) finish_kernel(const float* __restrict__ part,
                                                                   T* __restrict__ out, int cols,
                                                                   int slices) {
  __shared__ float sums[kFinishWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (c < cols)
    for (int i = warp; i < slices; i += kFinishWarps * kFinishUnroll) {
      float v[kFinishUnroll];
#pragma unroll
      for (int u = 0; u < kFinishUnroll; ++u) {
        const int j = i + u * kFinishWarps;
        v[u] = j < slices ? part[(int64_t)j * cols + c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < kFinishUnroll; ++u) s += v[u];
    }
  sums[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < cols) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kFinishWarps; ++w) t += sums[w][lane];
    out[c] = from_f<T>(t);
  }
}

template <class T>
int run(const void* in, void* out, int64_t rows, int cols, void* scratch, cudaStream_t stream) {
  const Split s = split_rows(rows, cols);
  const dim3 grid((cols + kBlockCols - 1) / kBlockCols, s.slices);
  partial_kernel<T><<<grid, kWarps * 32, 0, stream>>>((const T*)in, (float*)scratch, rows, cols, s.rows_per);
  B200NA_CUDA_TRY(cudaGetLastError());
  finish_kernel<T><<<(cols + 31) / 32, kFinishWarps * 32, 0, stream>>>((const float*)scratch, (T*)out, cols, s.slices);
  B200NA_CUDA_TRY(cudaGetLastError());
  return B200NA_OK;
}

}  // namespace
}  // namespace b200na

extern "C" B200NA_API int64_t b200na_column_sum_scratch(int64_t rows, int cols) {
  if (rows < 1 || cols < 1) return 0;
  return (int64_t)b200na::split_rows(rows, cols).slices * cols * (int64_t)sizeof(float);
}

extern "C" B200NA_API int b200na_column_sum(const void* in, void* out, int64_t rows, int cols, int dtype,
                                            void* scratch, b200na_stream_t stream) {
  using namespace b200na;
  if (!in || !out || !scratch || rows < 1 || cols < 1) return B200NA_ERR_INVALID_ARGUMENT;
  if (cols % 8 != 0 || reinterpret_cast<uintptr_t>(in) % 16 != 0) return B200NA_ERR_ALIGNMENT;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == B200NA_F16) return run<__half>(in, out, rows, cols, scratch, s);
  if (dtype == B200NA_BF16) return run<__nv_bfloat16>(in, out, rows, cols, scratch, s);
  return B200NA_ERR_UNSUPPORTED;
}
