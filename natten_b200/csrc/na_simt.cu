// Neighborhood attention forward on the ORIGINAL token layout with CUDA-core fp32 arithmetic
// (sm_100a). This is the path for fp32 operands and for head dims the tensor-core kernel does not
// take; it also accepts fp16/bf16 operands (converted to fp32 on load).
//
// Semantics follow the reference's naive kernel and mask
// (csrc/include/natten/cuda/reference/fna_reference_forward.hpp:63-211, mask.hpp:47-89, 220-225,
// 306-343): scaled logits, running max, exp, O = sum(p v) / sum(p), LSE = log(sum) + max, extra KV
// tokens attended by every query.
//
// A block owns 32 queries of one head and streams the keys of their windows' union past them (see
// simt_tile.cuh for the split and its reasons): S = Q K^T in 4 x 4 register tiles, online softmax
// per 64 keys with the 16 lanes that share a row, P through shared memory (read back by the same
// warp only), O accumulated in registers.
//
// Bound: the fp32 pipe on the union boxes, 2-3 times the attended pairs for small windows; for one
// small map (32 x 32, 128 blocks) the latency of a few dependent steps.
#include <math.h>

#include <mutex>
#include <unordered_set>

#include "common.cuh"
#include "simt_tile.cuh"

namespace b200na {
namespace {

using namespace simt;

template <int DM>
struct FwdSmem {
  float q[kRows * (DM + 4)];
  float k[kCols * (DM + 4)];
  float v[kCols * (DM + 4)];
  float w[kRows * kPStride];
  Cols cols[2];
  Rows rows;
};

template <class T>
struct FwdTensors {
  const T *q, *k, *v;
  T* o;
  float* lse;
  const T *add_k, *add_v;
};

// One item: the block's 32 queries, decoded in sm.rows and loaded in sm.q, against their keys. False if
// the sums are not finite and nothing was stored; kAgain: stored in any case (see simt_tile.cuh).
template <class T, int DM, bool kVec, bool kAgain>
__device__ __forceinline__ bool attend(FwdSmem<DM>& sm, const FwdTensors<T>& x, const Params& p) {
  const int tid = threadIdx.x;
  const int rg = tid >> 4, cl = tid & 15;
  const int nd = p.ax.ndim;
  const int dp = (p.D + 3) & ~3;
  const int64_t n_tok = (int64_t)sm.rows.box_len[0] * sm.rows.box_len[1] * sm.rows.box_len[2];
  const int64_t n_all = n_tok > 0 ? n_tok + p.n_extra : 0;   // no columns: padding rows only
  if (tid < kCols) decode_col<false>(p, sm.rows, n_tok, n_all, tid, sm.cols[0], tid);
  if (!kAgain) load_rows<T, DM, kVec, kRows>(sm.q, x.q, sm.rows.row, p.D);

  float m[4], sum[4], acc[4][OutCols<DM>::kPer];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    m[r] = -INFINITY;
    sum[r] = 0.f;
#pragma unroll
    for (int t = 0; t < OutCols<DM>::kPer; ++t) acc[r][t] = 0.f;
  }
  int buf = 0;
  for (int64_t j0 = 0; j0 < n_all; j0 += kCols, buf ^= 1) {
    __syncthreads();               // this step's column table is written, the last tiles are read
    const Cols& cols = sm.cols[buf];
    load_key_values<T, DM, kVec>(p, sm.rows, cols, j0, n_tok, n_all, sm.k, sm.v, x.k, x.v, x.add_k,
                                 x.add_v);
    if (tid < kCols && j0 + kCols < n_all)
      decode_col<false>(p, sm.rows, n_tok, n_all, j0 + kCols + tid, sm.cols[buf ^ 1], tid);
    __syncthreads();

    float s[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[r][i] = 0.f;
    dot_tile<DM>(sm.q, sm.k, rg, cl, dp, s);
    int4 cc[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) cc[i] = cols.c[cl + 16 * i];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float mx = -INFINITY;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s[r][i] = pair_on(sm.rows, rg * 4 + r, cc[i], nd) ? s[r][i] * p.scale : -INFINITY;
        mx = fmaxf(mx, s[r][i]);
      }
      const float m_new = fmaxf(m[r], row_max(mx));
      // a row without a key so far keeps -inf; its exponents must not become NaN
      const float ref = m_new == -INFINITY ? 0.f : m_new;
      const float corr = expf(m[r] - ref);      // exp(-inf) = 0 on the first keys
      float part = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float pj = expf(s[r][i] - ref);
        part += pj;
        sm.w[(rg * 4 + r) * kPStride + cl + 16 * i] =
            kAgain ? weight_if(pair_on(sm.rows, rg * 4 + r, cc[i], nd), pj) : pj;
      }
      sum[r] = sum[r] * corr + row_sum(part);
      m[r] = m_new;
#pragma unroll
      for (int t = 0; t < OutCols<DM>::kPer; ++t) acc[r][t] *= corr;
    }
    __syncwarp();                  // P rows are read by the warp that wrote them
    const int n4 = (int)min((int64_t)kCols, (n_all - j0 + 3) & ~(int64_t)3);
    if constexpr (kAgain) accumulate_interacting<DM>(sm.w, sm.v, rg, cl, n4, acc);
    else accumulate_tile<DM>(sm.w, sm.v, rg, cl, n4, acc);
  }
  if (!kAgain && __syncthreads_or(any_non_finite(acc))) return false;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t row = sm.rows.row[rg * 4 + r];
    if (row < 0) continue;
    store_row<T, DM>(x.o + row * p.D, acc[r], 1.f / sum[r], cl, p.D);
    if (x.lse && cl == 0) x.lse[row] = logf(sum[r]) + m[r];
  }
  return true;
}
template <class T, int DM, bool kVec>
__device__ __noinline__ void attend_again(FwdSmem<DM>& sm, const FwdTensors<T>& x, const Params& p) {
  attend<T, DM, kVec, true>(sm, x, p);
}

template <class T, int DM, bool kVec>
__global__ void __launch_bounds__(kThreads, fwd_blocks(DM)) na_simt_kernel(
    const __grid_constant__ FwdTensors<T> x, const __grid_constant__ Params p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  FwdSmem<DM>& sm = *reinterpret_cast<FwdSmem<DM>*>(smem_raw);
  for (int64_t item = blockIdx.x; item < p.n_items; item += gridDim.x) {
    __syncthreads();                 // the previous item's readers are done
    if (threadIdx.x < kRows) decode_rows<false>(p, item, sm.rows);
    __syncthreads();
    if (!attend<T, DM, kVec, false>(sm, x, p)) attend_again<T, DM, kVec>(sm, x, p);
  }
}

template <class T, int DM>
int launch_dm(const void* q, const void* k, const void* v, void* o, float* lse, const void* ak,
              const void* av, Params& p, cudaStream_t stream) {
  const bool vec = vectorised(p.D, sizeof(T), reinterpret_cast<uintptr_t>(q) |
                              reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v));
  const void* fn = vec ? (const void*)na_simt_kernel<T, DM, true>
                       : (const void*)na_simt_kernel<T, DM, false>;
  FwdTensors<T> x = {(const T*)q, (const T*)k, (const T*)v, (T*)o, lse, (const T*)ak, (const T*)av};
  void* args[] = {(void*)&x, (void*)&p};
  return simt::launch(fn, p.n_items, (int)sizeof(FwdSmem<DM>), args, stream);
}
template <class T>
int launch_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const void* ak,
               const void* av, Params& p, cudaStream_t stream) {
  plan_rows(p);
  if (p.D <= 32) return launch_dm<T, 32>(q, k, v, o, lse, ak, av, p, stream);
  if (p.D <= 64) return launch_dm<T, 64>(q, k, v, o, lse, ak, av, p, stream);
  if (p.D <= 128) return launch_dm<T, 128>(q, k, v, o, lse, ak, av, p, stream);
  return launch_dm<T, 256>(q, k, v, o, lse, ak, av, p, stream);
}
int launch_typed(const void* q, const void* k, const void* v, void* o, float* lse, const void* ak,
                 const void* av, Params& p, int dtype, cudaStream_t s) {
  switch (dtype) {
    case B200NA_F32: return launch_fwd<float>(q, k, v, o, lse, ak, av, p, s);
    case B200NA_F16: return launch_fwd<__half>(q, k, v, o, lse, ak, av, p, s);
    case B200NA_BF16: return launch_fwd<__nv_bfloat16>(q, k, v, o, lse, ak, av, p, s);
    default: return B200NA_ERR_INVALID_ARGUMENT;
  }
}

}  // namespace

namespace simt {
int launch(const void* fn, int64_t items, int smem_bytes, void** args, cudaStream_t stream) {
  if (smem_bytes > 48 * 1024) {
    static std::mutex mu;
    static std::unordered_set<const void*> done[64];
    int dev = 0;
    B200NA_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B200NA_ERR_DEVICE;
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev].count(fn) == 0) {
      B200NA_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           smem_bytes));
      done[dev].insert(fn);
    }
  }
  if (items == 0) return B200NA_OK;
  const int64_t grid = items < 0x7fffffff ? items : 0x7fffffff;
  B200NA_CUDA_TRY(cudaLaunchKernel(fn, dim3((unsigned)grid), dim3(kThreads), args, smem_bytes, stream));
  return B200NA_OK;
}
}  // namespace simt

// Dense attention on CUDA cores (fp32 operands, or head dims the tensor-core kernel does not
// take); called by b200na_fmha_forward.
int simt_dense_forward(const void* q, const void* k, const void* v, void* o, float* lse, int B,
                       int Nq, int Nk, int Hq, int Hkv, int D, int dtype, float scale, int causal,
                       cudaStream_t stream) {
  if (D > kMaxD) return B200NA_ERR_UNSUPPORTED;
  Params p;
  memset(&p, 0, sizeof(p));
  p.ax.ndim = 1;
  for (int a = 0; a < B200NA_MAX_DIM; ++a) {
    p.ax.shape[a] = 1; p.ax.kernel[a] = 1; p.ax.stride[a] = 1; p.ax.dilation[a] = 1;
  }
  p.ax.shape[0] = Nk;
  p.ax.causal[0] = causal ? 1 : 0;
  p.N = Nk; p.Nq = Nq; p.dense = 1; p.G = 1;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.row_heads = Hq; p.D = D; p.scale = scale;
  return launch_typed(q, k, v, o, lse, nullptr, nullptr, p, dtype, stream);
}

}  // namespace b200na

extern "C" B200NA_API int b200na_na_forward_simt(const void* q, const void* k, const void* v, void* o,
                                      float* lse, int ndim, const int* shape, const int* kernel,
                                      const int* stride, const int* dilation, const int* causal,
                                      int B, int Hq, int Hkv, int D, int dtype, float scale,
                                      const void* add_k, const void* add_v, int n_extra,
                                      b200na_stream_t stream) {
  using namespace b200na;
  if (!q || !k || !v || !o) return B200NA_ERR_INVALID_ARGUMENT;
  if (B < 1 || Hq < 1 || Hkv < 1 || Hq % Hkv != 0 || D < 1) return B200NA_ERR_INVALID_ARGUMENT;
  if (D > simt::kMaxD) return B200NA_ERR_UNSUPPORTED;
  if (n_extra < 0 || (n_extra > 0 && (!add_k || !add_v))) return B200NA_ERR_INVALID_ARGUMENT;
  simt::Params p;
  memset(&p, 0, sizeof(p));
  int rc = fill_axes(p.ax, ndim, shape, kernel, stride, dilation, causal);
  if (rc != B200NA_OK) return rc;
  p.N = 1;
  int64_t groups = 1;
  for (int a = 0; a < ndim; ++a) {
    p.N *= shape[a];
    groups *= p.ax.dilation[a];
  }
  if (groups > 0x7fffffffLL) return B200NA_ERR_UNSUPPORTED;
  p.G = (int)groups;
  p.Nq = p.N;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.row_heads = Hq; p.D = D; p.n_extra = n_extra; p.scale = scale;
  return launch_typed(q, k, v, o, lse, add_k, add_v, p, dtype, reinterpret_cast<cudaStream_t>(stream));
}
