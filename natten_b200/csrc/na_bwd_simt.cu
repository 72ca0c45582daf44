// Neighborhood attention BACKWARD on the original token layout with CUDA-core fp32 arithmetic
// (sm_100a): dQ, dK, dV (and the gradients of extra key/value tokens) for fp32 / fp16 / bf16
// operands and any head dim up to 256. Companion of na_simt.cu (same tiles, simt_tile.cuh).
//
// Semantics follow the reference's naive backward kernels
// (csrc/include/natten/cuda/reference/fna_reference_backward.hpp:62-160 dQ, 177-275 dK, 293-385 dV)
// and its delta pre-pass (csrc/src/compute_delta.cu): with s_ij = scale q_i.k_j,
// P_ij = exp(s_ij - LSE_i), dP_ij = dO_i.v_j, delta_i = dO_i.O_i,
//   dS_ij = scale P_ij (dP_ij - delta_i),  dQ_i = sum_j dS_ij k_j,
//   dK_j = sum_i dS_ij q_i,  dV_j = sum_i P_ij dO_i.
// Two kernels, no atomics, deterministic:
//   * dQ: a block's rows are 32 queries, the columns their windows' keys. It also computes delta of
//     its rows (dO is in shared memory anyway) and leaves it for the second kernel.
//   * dK/dV: the rows are 32 keys, the columns the queries that attend them - a box too, because
//     window start and end are monotone in the query coordinate. Extra tokens are attended by every
//     query: the same kernel with the whole layout as the box.
// Bound: the fp32 pipe (3 products in the first kernel, 4 in the second, on the union boxes).
#include <math.h>

#include "common.cuh"
#include "fna_host.cuh"
#include "simt_tile.cuh"

namespace b200na {
namespace {

using namespace simt;

template <int DM, bool kKeyRows>
struct BwdSmem {
  float r1[kRows * (DM + 4)];     // rows: Q, dO or K, V
  float r2[kRows * (DM + 4)];
  float c1[kCols * (DM + 4)];     // columns: K, V or Q, dO
  float c2[kCols * (DM + 4)];
  float ds[kRows * kPStride];
  float pr[kKeyRows ? kRows * kPStride : 4];
  Cols cols[2];
  float lse[kCols], delta[kCols];   // of the columns (dK/dV)
  Rows rows;
};

// out0 = dQ or dK, out1 = dV.
template <class T>
struct BwdTensors {
  const T *q, *k, *v, *o, *d_out;
  const float* lse;
  float* delta;
  const T *add_k, *add_v;
  T *out0, *out1;
};

// One item: the block's 32 rows, decoded in sm.rows, against their columns. False if the sums are not
// finite and nothing was stored; kAgain: stored in any case (see simt_tile.cuh).
template <class T, int DM, bool kVec, bool kKeyRows, bool kAgain>
__device__ __forceinline__ bool gradients(BwdSmem<DM, kKeyRows>& sm, const BwdTensors<T>& x,
                                          const Params& p) {
  const int tid = threadIdx.x;
  const int rg = tid >> 4, cl = tid & 15;
  const int nd = p.ax.ndim;
  const int dp = (p.D + 3) & ~3;
  int64_t n_tok = (int64_t)sm.rows.box_len[0] * sm.rows.box_len[1] * sm.rows.box_len[2];
  int64_t n_all = n_tok;
  if (kKeyRows) n_all = n_tok = n_tok * (p.Hq / p.Hkv);
  else if (n_tok > 0) n_all += p.n_extra;
  if (tid < kCols) decode_col<kKeyRows>(p, sm.rows, n_tok, n_all, tid, sm.cols[0], tid);
  float row_lse[4], row_delta[4];
  if (kKeyRows) {
    load_rows<T, DM, kVec, kRows>(sm.r1, p.extra_rows ? x.add_k : x.k, sm.rows.row, p.D);
    load_rows<T, DM, kVec, kRows>(sm.r2, p.extra_rows ? x.add_v : x.v, sm.rows.row, p.D);
  } else {
    load_rows<T, DM, kVec, kRows>(sm.r1, x.q, sm.rows.row, p.D);
    load_rows<T, DM, kVec, kRows>(sm.r2, x.d_out, sm.rows.row, p.D);
    load_rows<T, DM, kVec, kRows>(sm.c1, x.o, sm.rows.row, p.D);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t row = sm.rows.row[rg * 4 + r];
      float part = 0.f;
      for (int d = cl; d < p.D; d += 16)
        part = fmaf(sm.r2[(rg * 4 + r) * (DM + 4) + d], sm.c1[(rg * 4 + r) * (DM + 4) + d], part);
      row_delta[r] = row_sum(part);
      row_lse[r] = row >= 0 ? x.lse[row] : 0.f;
      if (row >= 0 && cl == 0) x.delta[row] = row_delta[r];
    }
  }

  float acc0[4][OutCols<DM>::kPer], acc1[4][kKeyRows ? OutCols<DM>::kPer : 1];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int t = 0; t < OutCols<DM>::kPer; ++t) {
      acc0[r][t] = 0.f;
      acc1[r][kKeyRows ? t : 0] = 0.f;
    }
  int buf = 0;
  for (int64_t j0 = 0; j0 < n_all; j0 += kCols, buf ^= 1) {
    __syncthreads();               // this step's column table is written, the last tiles are read
    const Cols& cols = sm.cols[buf];
    if (kKeyRows) {
      load_rows<T, DM, kVec, kCols>(sm.c1, x.q, cols.row, p.D);
      load_rows<T, DM, kVec, kCols>(sm.c2, x.d_out, cols.row, p.D);
      if (tid < kCols) {
        const int64_t row = cols.row[tid];
        sm.lse[tid] = row >= 0 ? x.lse[row] : 0.f;
        sm.delta[tid] = row >= 0 ? x.delta[row] : 0.f;
      }
    } else {
      load_key_values<T, DM, kVec>(p, sm.rows, cols, j0, n_tok, n_all, sm.c1, sm.c2, x.k, x.v,
                                   x.add_k, x.add_v);
    }
    if (tid < kCols && j0 + kCols < n_all)
      decode_col<kKeyRows>(p, sm.rows, n_tok, n_all, j0 + kCols + tid, sm.cols[buf ^ 1], tid);
    __syncthreads();

    float s[4][4], dpv[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[r][i] = dpv[r][i] = 0.f;
    dot_tile<DM>(sm.r1, sm.c1, rg, cl, dp, s);
    dot_tile<DM>(sm.r2, sm.c2, rg, cl, dp, dpv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int4 cc = cols.c[cl + 16 * i];
      const float cl_lse = kKeyRows ? sm.lse[cl + 16 * i] : 0.f;
      const float cl_delta = kKeyRows ? sm.delta[cl + 16 * i] : 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool on = pair_on(sm.rows, rg * 4 + r, cc, nd);
        const float pj = on ? expf(s[r][i] * p.scale - (kKeyRows ? cl_lse : row_lse[r])) : 0.f;
        const float ds = p.scale * pj * (dpv[r][i] - (kKeyRows ? cl_delta : row_delta[r]));
        const int at = (rg * 4 + r) * kPStride + cl + 16 * i;
        sm.ds[at] = kAgain ? weight_if(on, ds) : ds;
        if (kKeyRows) sm.pr[at] = kAgain ? weight_if(on, pj) : pj;
      }
    }
    __syncwarp();                  // these rows are read by the warp that wrote them
    const int n4 = (int)min((int64_t)kCols, (n_all - j0 + 3) & ~(int64_t)3);
    if constexpr (kAgain) {
      accumulate_interacting<DM>(sm.ds, sm.c1, rg, cl, n4, acc0);
      if constexpr (kKeyRows) accumulate_interacting<DM>(sm.pr, sm.c2, rg, cl, n4, acc1);
    } else {
      accumulate_tile<DM>(sm.ds, sm.c1, rg, cl, n4, acc0);
      if constexpr (kKeyRows) accumulate_tile<DM>(sm.pr, sm.c2, rg, cl, n4, acc1);
    }
  }
  if (!kAgain && __syncthreads_or(any_non_finite(acc0) || any_non_finite(acc1))) return false;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int64_t row = sm.rows.row[rg * 4 + r];
    if (row < 0) continue;
    store_row<T, DM>(x.out0 + row * p.D, acc0[r], 1.f, cl, p.D);
    if constexpr (kKeyRows) store_row<T, DM>(x.out1 + row * p.D, acc1[r], 1.f, cl, p.D);
  }
  return true;
}
template <class T, int DM, bool kVec, bool kKeyRows>
__device__ __noinline__ void gradients_again(BwdSmem<DM, kKeyRows>& sm, const BwdTensors<T>& x,
                                             const Params& p) {
  gradients<T, DM, kVec, kKeyRows, true>(sm, x, p);
}

// Whether a thread's share of the block's results, as another kernel left them, holds a NaN or an infinity
// (16-bit types, D a multiple of 8, 16-byte aligned).
template <class T, bool kKeyRows>
__device__ __forceinline__ bool non_finite_results(const BwdTensors<T>& x, const Rows& s, int D) {
  float t = 0.f;
  if constexpr (sizeof(T) == 2) {
    const int chunks = D / 8;
    for (int i = threadIdx.x; i < kRows * chunks; i += kThreads) {
      const int64_t row = s.row[i / chunks];
      if (row < 0) continue;
#pragma unroll
      for (int o = 0; o < (kKeyRows ? 2 : 1); ++o) {
        const uint4 v = *reinterpret_cast<const uint4*>((o ? x.out1 : x.out0) + row * D + i % chunks * 8);
        const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
        for (int k = 0; k < 8; ++k) t = fmaf(ldf(e + k), 0.f, t);
      }
    }
  }
  return t != 0.f;   // NaN
}

template <class T, int DM, bool kVec, bool kKeyRows>
__global__ void __launch_bounds__(kThreads, bwd_blocks(DM)) na_bwd_kernel(
    const __grid_constant__ BwdTensors<T> x, const __grid_constant__ Params p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  using SM = BwdSmem<DM, kKeyRows>;
  SM& sm = *reinterpret_cast<SM*>(smem_raw);
  if (p.redo && *p.redo == 0) return;
  for (int64_t item = blockIdx.x; item < p.n_items; item += gridDim.x) {
    __syncthreads();                 // the previous item's readers are done
    if (threadIdx.x < kRows) decode_rows<kKeyRows>(p, item, sm.rows);
    __syncthreads();
    if (p.redo && !__syncthreads_or(non_finite_results<T, kKeyRows>(x, sm.rows, p.D))) continue;
    if (!gradients<T, DM, kVec, kKeyRows, false>(sm, x, p)) gradients_again<T, DM, kVec, kKeyRows>(sm, x, p);
  }
}

struct BwdPointers {
  const void *q, *k, *v, *o, *d_out;
  const float* lse;
  const void *add_k, *add_v;
  void *dq, *dk, *dv, *d_add_k, *d_add_v;
  float* delta;
};

template <class T, int DM>
int launch_bwd_dm(BwdPointers& a, const Params& base, cudaStream_t stream) {
  const bool vec = vectorised(base.D, sizeof(T),
                              reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) |
                              reinterpret_cast<uintptr_t>(a.v) | reinterpret_cast<uintptr_t>(a.o) |
                              reinterpret_cast<uintptr_t>(a.d_out) |
                              reinterpret_cast<uintptr_t>(a.add_k) |
                              reinterpret_cast<uintptr_t>(a.add_v));
  const void* fn_q = vec ? (const void*)na_bwd_kernel<T, DM, true, false>
                         : (const void*)na_bwd_kernel<T, DM, false, false>;
  const void* fn_k = vec ? (const void*)na_bwd_kernel<T, DM, true, true>
                         : (const void*)na_bwd_kernel<T, DM, false, true>;
  // every query interacts with every extra token: nothing reaches their sums that does not belong there
  for (int pass = 0; pass < (base.n_extra > 0 && !base.redo ? 3 : 2); ++pass) {
    Params p = base;
    p.row_heads = pass == 0 ? p.Hq : p.Hkv;
    if (pass == 2) {   // extra tokens: every query is a column, dilation groups do not matter
      p.extra_rows = 1;
      p.G = 1;
      for (int x = 0; x < B200NA_MAX_DIM; ++x) p.ax.dilation[x] = 1;
    }
    plan_rows(p);
    BwdTensors<T> x = {(const T*)a.q, (const T*)a.k, (const T*)a.v, (const T*)a.o,
                       (const T*)a.d_out, a.lse, a.delta, (const T*)a.add_k, (const T*)a.add_v,
                       (T*)(pass == 0 ? a.dq : (pass == 1 ? a.dk : a.d_add_k)),
                       (T*)(pass == 0 ? nullptr : (pass == 1 ? a.dv : a.d_add_v))};
    void* args[] = {(void*)&x, (void*)&p};
    // a look at *redo is all there is to do nearly always: as many blocks as are resident at once
    const int64_t blocks = p.redo ? min(p.n_items, (int64_t)148 * bwd_blocks(DM)) : p.n_items;
    const int rc = simt::launch(pass == 0 ? fn_q : fn_k, blocks,
                                (int)(pass == 0 ? sizeof(BwdSmem<DM, false>)
                                                : sizeof(BwdSmem<DM, true>)), args, stream);
    if (rc != B200NA_OK) return rc;
  }
  return B200NA_OK;
}
template <class T>
int launch_bwd(BwdPointers& a, const Params& p, cudaStream_t stream) {
  if (p.D <= 32) return launch_bwd_dm<T, 32>(a, p, stream);
  if (p.D <= 64) return launch_bwd_dm<T, 64>(a, p, stream);
  if (p.D <= 128) return launch_bwd_dm<T, 128>(a, p, stream);
  return launch_bwd_dm<T, 256>(a, p, stream);
}

// delta[row] = sum_d dO * O for the tensor-core backward: kLanes (a power of two) lanes per row of
// `chunks` <= kLanes 16-byte pieces.
constexpr int kDeltaThreads = 256;
template <class T, int kLanes>
__global__ void __launch_bounds__(kDeltaThreads) delta_kernel(const T* __restrict__ o,
                                                              const T* __restrict__ d_out,
                                                              float* __restrict__ delta,
                                                              int64_t rows, int chunks, int vec) {
  const int64_t i = (int64_t)blockIdx.x * kDeltaThreads + threadIdx.x;
  const int64_t row = i / kLanes;
  const int ch = (int)(i % kLanes);
  float acc = 0.f;
  if (row < rows && ch < chunks) {
    const int64_t at = (row * chunks + ch) * 8;
    if (vec) {
      const uint4 x = *reinterpret_cast<const uint4*>(o + at),
                  y = *reinterpret_cast<const uint4*>(d_out + at);
      const T* a = reinterpret_cast<const T*>(&x);
      const T* b = reinterpret_cast<const T*>(&y);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc = fmaf(ldf(a + e), ldf(b + e), acc);
    } else {   // o need not be 16-byte aligned
      for (int e = 0; e < 8; ++e) acc = fmaf(ldf(o + at + e), ldf(d_out + at + e), acc);
    }
  }
#pragma unroll
  for (int off = kLanes / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (row < rows && ch == 0) delta[row] = acc;
}
template <class T>
int launch_delta_typed(const void* o, const void* d_out, float* delta, int64_t rows, int D,
                       cudaStream_t stream) {
  const int chunks = D / 8;
  int lanes = 1;
  while (lanes < chunks) lanes <<= 1;
  const int64_t blocks = (rows * lanes + kDeltaThreads - 1) / kDeltaThreads;
  if (blocks > 0x7fffffff || lanes > 16) return B200NA_ERR_UNSUPPORTED;
  const int vec = (reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(d_out)) % 16 == 0;
#define B200NA_DELTA(L)                                                       \
  case L:                                                                     \
    delta_kernel<T, L><<<(unsigned)blocks, kDeltaThreads, 0, stream>>>(       \
        (const T*)o, (const T*)d_out, delta, rows, chunks, vec);              \
    break
  switch (lanes) {
    B200NA_DELTA(1);
    B200NA_DELTA(2);
    B200NA_DELTA(4);
    B200NA_DELTA(8);
    B200NA_DELTA(16);
  }
#undef B200NA_DELTA
  B200NA_CUDA_TRY(cudaGetLastError());
  return B200NA_OK;
}

// A lane per 16 bytes, kLanes per row, a block's largest row in one atomic. Squared norms are not negative,
// so that their bits order like they do, with NaN above all.
template <int kLanes>
__global__ void __launch_bounds__(kDeltaThreads) max_norms_kernel(NormRows a, NormRows b, NormRows c,
                                                                  int chunks, unsigned* norms) {
  const NormRows in = blockIdx.y == 0 ? a : (blockIdx.y == 1 ? b : c);
  const int ch = threadIdx.x % kLanes;
  const int64_t rows = in.tokens * in.heads, step = (int64_t)gridDim.x * (kDeltaThreads / kLanes);
  unsigned most = 0;
  for (int64_t r0 = (int64_t)blockIdx.x * (kDeltaThreads / kLanes); r0 < rows; r0 += step) {
    const int64_t row = r0 + threadIdx.x / kLanes;
    float sum = 0.f;
    if (row < rows && ch < chunks) {
      const __half* p = static_cast<const __half*>(in.rows) + (row / in.heads) * in.token_stride +
                        (row % in.heads) * chunks * 8 + ch * 8;
      const uint4 x = *reinterpret_cast<const uint4*>(p);
      const __half* v = reinterpret_cast<const __half*>(&x);
#pragma unroll
      for (int e = 0; e < 8; ++e) sum = fmaf(ldf(v + e), ldf(v + e), sum);
    }
#pragma unroll
    for (int off = kLanes / 2; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    most = max(most, __float_as_uint(sum) & 0x7fffffffu);
  }
  most = __reduce_max_sync(0xffffffffu, most);
  __shared__ unsigned part[kDeltaThreads / 32];
  if (threadIdx.x % 32 == 0) part[threadIdx.x / 32] = most;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kDeltaThreads / 32; ++w) most = max(most, part[w]);
    atomicMax(norms + in.slot, most);
  }
}

}  // namespace

int launch_max_norms(const NormRows* in, int n_inputs, int D, float* norms, cudaStream_t stream) {
  if (n_inputs < 2 || n_inputs > 3 || D % 8 != 0 || D < 8 || D > 128) return B200NA_ERR_INVALID_ARGUMENT;
  const dim3 grid(148, n_inputs);
  const NormRows& last = in[n_inputs - 1];
  unsigned* out = reinterpret_cast<unsigned*>(norms);
  if (D <= 64) max_norms_kernel<8><<<grid, kDeltaThreads, 0, stream>>>(in[0], in[1], last, D / 8, out);
  else max_norms_kernel<16><<<grid, kDeltaThreads, 0, stream>>>(in[0], in[1], last, D / 8, out);
  B200NA_CUDA_TRY(cudaGetLastError());
  return B200NA_OK;
}

int launch_delta(const void* o, const void* d_out, float* delta, int64_t rows, int D, int dtype,
                 cudaStream_t stream) {
  // the tensor-core backward takes 16-bit operands, head dims that are multiples of 8
  if (dtype == B200NA_F16) return launch_delta_typed<__half>(o, d_out, delta, rows, D, stream);
  if (dtype == B200NA_BF16) return launch_delta_typed<__nv_bfloat16>(o, d_out, delta, rows, D, stream);
  return B200NA_ERR_INVALID_ARGUMENT;
}

int simt_backward(
    const void* q, const void* k, const void* v, const void* o, const void* d_out, const float* lse,
    const void* add_k, const void* add_v, int n_extra, void* dq, void* dk, void* dv, void* d_add_k,
    void* d_add_v, float* delta_scratch, int ndim, const int* shape, const int* kernel,
    const int* stride, const int* dilation, const int* causal, int B, int Hq, int Hkv, int D,
    int dtype, float scale, const unsigned* redo, cudaStream_t stream) {
  if (!q || !k || !v || !o || !d_out || !lse || !dq || !dk || !dv || !delta_scratch)
    return B200NA_ERR_INVALID_ARGUMENT;
  if (n_extra < 0 || (n_extra > 0 && (!add_k || !add_v || !d_add_k || !d_add_v)))
    return B200NA_ERR_INVALID_ARGUMENT;
  if (B < 1 || Hq < 1 || Hkv < 1 || Hq % Hkv != 0 || D < 1 || !(scale > 0.f))
    return B200NA_ERR_INVALID_ARGUMENT;
  if (D > simt::kMaxD) return B200NA_ERR_UNSUPPORTED;
  simt::Params p;
  memset(&p, 0, sizeof(p));
  int rc = fill_axes(p.ax, ndim, shape, kernel, stride, dilation, causal);
  if (rc != B200NA_OK) return rc;
  p.N = 1;
  int64_t groups = 1;
  for (int a = 0; a < ndim; ++a) {
    p.N *= p.ax.shape[a];
    groups *= p.ax.dilation[a];
  }
  if (groups > 0x7fffffffLL) return B200NA_ERR_UNSUPPORTED;
  p.G = (int)groups;
  p.Nq = p.N;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.D = D;
  p.n_extra = n_extra;
  p.scale = scale;
  p.redo = redo;
  BwdPointers a = {q, k, v, o, d_out, lse, add_k, add_v, dq, dk, dv, d_add_k, d_add_v, delta_scratch};
  switch (dtype) {
    case B200NA_F32: return launch_bwd<float>(a, p, stream);
    case B200NA_F16: return launch_bwd<__half>(a, p, stream);
    case B200NA_BF16: return launch_bwd<__nv_bfloat16>(a, p, stream);
    default: return B200NA_ERR_INVALID_ARGUMENT;
  }
}
}  // namespace b200na

extern "C" B200NA_API int b200na_na_backward_simt(
    const void* q, const void* k, const void* v, const void* o, const void* d_out, const float* lse,
    const void* add_k, const void* add_v, int n_extra, void* dq, void* dk, void* dv, void* d_add_k,
    void* d_add_v, float* delta_scratch, int ndim, const int* shape, const int* kernel,
    const int* stride, const int* dilation, const int* causal, int B, int Hq, int Hkv, int D,
    int dtype, float scale, b200na_stream_t stream) {
  return b200na::simt_backward(q, k, v, o, d_out, lse, add_k, add_v, n_extra, dq, dk, dv, d_add_k, d_add_v,
                               delta_scratch, ndim, shape, kernel, stride, dilation, causal, B, Hq, Hkv, D,
                               dtype, scale, nullptr, reinterpret_cast<cudaStream_t>(stream));
}
