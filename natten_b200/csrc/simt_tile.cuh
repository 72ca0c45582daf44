// Device pieces shared by the CUDA-core attention kernels (na_simt.cu forward, na_bwd_simt.cu
// backward): a block of 128 threads owns 32 ROWS (a box of queries, or of keys) of one head and
// streams the COLUMNS those rows interact with past them, 64 at a time.
//
// Why tiles: with one warp per row every key and value is read from L1 / L2 once per query and
// every product waits for a load. In a tile each column is fetched once for 32 rows, the products
// run from shared memory with a 4 x 4 register tile per thread (8 16-byte shared loads per 64 FMA
// instructions), and the fp32 pipe is the bound. 32 rows because windows are small: the union of
// the windows of a 4 x 8 box is 2-3 times one window, that of 64 or 128 rows far more, and small
// maps still give enough blocks to fill the chip.
//
// Columns are enumerated linearly inside the union box of the rows' spans (no column tile shape, no
// padding except in the last 64), extra tokens after them. All sums are fp32 FMA.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace b200na {
namespace simt {

constexpr int kRows = 32;      // rows of a block
constexpr int kCols = 64;      // columns per step
constexpr int kThreads = 128;
constexpr int kPStride = kCols + 4;
constexpr int kMaxD = 256;
// Blocks per SM of the kernels for head dims up to DM, the registers' share: as many as the shared memory
// lets in where that is few, so that the function for non-finite columns (accumulate_interacting), which
// is rarely called, does not raise the registers of all.
constexpr int fwd_blocks(int DM) { return DM <= 32 ? 5 : (DM <= 64 ? 4 : (DM <= 128 ? 2 : 1)); }
constexpr int bwd_blocks(int DM) { return DM <= 32 ? 4 : (DM <= 64 ? 3 : 1); }

template <class T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<__half>(const __half* p) { return __half2float(*p); }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) {
  return __bfloat162float(*p);
}
template <class T> __device__ __forceinline__ void stf(T* p, float v);
template <> __device__ __forceinline__ void stf<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void stf<__half>(__half* p, float v) { *p = __float2half_rn(v); }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float v) {
  *p = __float2bfloat16_rn(v);
}
template <class T> __device__ __forceinline__ float4 ldf4(const T* p);
template <> __device__ __forceinline__ float4 ldf4<float>(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}
template <> __device__ __forceinline__ float4 ldf4<__half>(const __half* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x)),
               b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
template <> __device__ __forceinline__ float4 ldf4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x)),
               b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

struct Params {
  NaAxes ax;
  int64_t N;          // key/value tokens per batch entry
  int64_t Nq;         // query tokens per batch entry (== N except for dense cross attention)
  int dense;          // dense attention: every query sees keys [0, N) (causal: [0, i + 1))
  int extra_rows;     // backward: the rows are the n_extra tokens, the columns all queries
  const unsigned* redo;   // backward, not null: the results are there; if *redo is not 0, items with a
                          // result that is not finite are done again
  int G;              // dilation groups
  int T[B200NA_MAX_DIM];   // row tile shape, product kRows
  int R[B200NA_MAX_DIM];   // row tiles per axis of the largest dilation group
  int64_t n_items;    // row tiles x heads x batch x groups
  int row_heads;      // heads the rows carry
  int B, Hq, Hkv, D;
  int n_extra;
  float scale;
};

// Queries of one axis (dilation-group coordinates, extent L) whose window holds key coordinate j:
// [lo, hi). Window start and end never decrease with the query coordinate: two bisections.
__device__ __forceinline__ void attending_queries(int j, int k, int s, int L, int causal, int& lo,
                                                  int& hi) {
  int a = 0, b = L;
  while (a < b) {  // first query whose window end is beyond j
    const int mid = (a + b) >> 1;
    const int st = win_start(mid, k, s, L, causal);
    if (win_end(mid, st, k, L, causal) > j) b = mid; else a = mid + 1;
  }
  lo = a;
  b = L;
  while (a < b) {  // first query whose window start is beyond j
    const int mid = (a + b) >> 1;
    if (win_start(mid, k, s, L, causal) > j) b = mid; else a = mid + 1;
  }
  hi = a;
}

// What a block knows about its rows and their columns (shared memory).
struct Rows {
  int64_t row[kRows];                    // row index in the row tensors (heads included), -1: none
  int lo[kRows][B200NA_MAX_DIM];         // span of columns the row interacts with
  int len[kRows][B200NA_MAX_DIM];
  int box_lo[B200NA_MAX_DIM], box_len[B200NA_MAX_DIM];   // union of the spans
  int g[B200NA_MAX_DIM];                 // dilation group of the block
  int64_t b;
  int h;                                 // head of the rows
};
// A column: its row index in the column tensors, its coordinates, its kind.
enum : int { kNone = 0, kToken = 1, kExtra = 2 };
struct Cols {
  int4 c[kCols];                         // x, y, z coordinates, w kind
  int64_t row[kCols];                    // -1: none, or an extra token
};

// Filled by warp 0 (one lane per row).
template <bool kKeyRows>
__device__ __forceinline__ void decode_rows(const Params& p, int64_t item, Rows& s) {
  const int lane = threadIdx.x;
  const int nd = p.ax.ndim;
  int64_t tile = item, tiles = (int64_t)p.R[0] * p.R[1] * p.R[2];
  const int64_t rest = item / tiles;
  tile -= rest * tiles;
  const int64_t bp = rest / p.row_heads;
  const int h = (int)(rest - bp * p.row_heads);
  const int64_t b = bp / p.G;
  int gl = (int)(bp - b * p.G);
  int r = lane;
  int64_t tok = 0;
  bool valid = true;
  int tr[B200NA_MAX_DIM], tt[B200NA_MAX_DIM], gg[B200NA_MAX_DIM];
#pragma unroll
  for (int a = B200NA_MAX_DIM - 1; a >= 0; --a) {   // last axis fastest
    tr[a] = r % p.T[a]; r /= p.T[a];
    tt[a] = (int)(tile % p.R[a]); tile /= p.R[a];
    gg[a] = gl % p.ax.dilation[a]; gl /= p.ax.dilation[a];
  }
  int lo[B200NA_MAX_DIM], hi[B200NA_MAX_DIM];
#pragma unroll
  for (int a = 0; a < B200NA_MAX_DIM; ++a) {
    const int i = tt[a] * p.T[a] + tr[a];
    const int d = p.ax.dilation[a];
    lo[a] = 0; hi[a] = 1;
    if (kKeyRows && p.extra_rows) {
      if (a == 0) { valid = i < p.n_extra; tok = i; }
      hi[a] = p.ax.shape[a];
    } else if (p.dense) {
      if (a == 0) {
        valid = i < p.Nq;
        tok = i;
        hi[a] = p.ax.causal[0] ? (int)min((int64_t)i + 1, p.N) : (int)p.N;
      }
    } else if (a < nd) {
      const int L = group_extent(p.ax.shape[a], d, gg[a]);
      valid = valid && i < L;
      const int ic = imin(i, L - 1);
      if (kKeyRows) {
        attending_queries(ic, p.ax.kernel[a], p.ax.stride[a], L, p.ax.causal[a], lo[a], hi[a]);
      } else {
        lo[a] = win_start(ic, p.ax.kernel[a], p.ax.stride[a], L, p.ax.causal[a]);
        hi[a] = win_end(ic, lo[a], p.ax.kernel[a], L, p.ax.causal[a]);
      }
      tok = tok * p.ax.shape[a] + ((int64_t)i * d + gg[a]);
    }
  }
  const int64_t n_rows = kKeyRows && p.extra_rows ? p.n_extra : p.Nq;
  s.row[lane] = valid ? (b * n_rows + tok) * p.row_heads + h : -1;
#pragma unroll
  for (int a = 0; a < B200NA_MAX_DIM; ++a) {
    s.lo[lane][a] = lo[a];
    s.len[lane][a] = valid ? hi[a] - lo[a] : 0;
    const int bl = __reduce_min_sync(0xffffffffu, valid ? lo[a] : 0x7fffffff);
    const int bh = __reduce_max_sync(0xffffffffu, valid ? hi[a] : 0);
    if (lane == 0) {
      s.box_lo[a] = bl;
      s.box_len[a] = bh > bl ? bh - bl : 0;   // a block of padding rows has no columns
      s.g[a] = gg[a];
    }
  }
  if (lane == 0) { s.b = b; s.h = h; }
}

// Column number j (of the block's enumeration) into slot `slot`; one thread per slot. kKeyRows:
// the columns are the queries of the kv head's group, head after head.
template <bool kKeyRows>
__device__ __forceinline__ void decode_col(const Params& p, const Rows& s, int64_t n_tok,
                                           int64_t n_all, int64_t j, Cols& c, int slot) {
  int64_t row = -1;
  int4 cc = make_int4(0, 0, 0, kNone);
  if (j < n_tok) {
    const int rep = p.Hq / p.Hkv;
    int head = kKeyRows ? s.h * rep : s.h / rep;
    int64_t idx = j;
    const unsigned l1 = s.box_len[1], l2 = s.box_len[2];
    if (kKeyRows && rep > 1) {
      const int64_t per = (int64_t)s.box_len[0] * l1 * l2;
      const int hh = (int)(idx / per);
      idx -= hh * per;
      head += hh;
    }
    int64_t c0 = idx;
    unsigned c1 = 0, c2 = 0;
    if (p.ax.ndim > 1) {
      if (idx <= 0xffffffffll) {   // boxes are small: 32-bit divisions
        unsigned t = (unsigned)idx;
        c2 = t % l2; t /= l2;
        c1 = t % l1;
        c0 = t / l1;
      } else {
        c2 = (unsigned)(c0 % l2); c0 /= l2;
        c1 = (unsigned)(c0 % l1); c0 /= l1;
      }
    }
    const int x[B200NA_MAX_DIM] = {s.box_lo[0] + (int)c0, s.box_lo[1] + (int)c1,
                                   s.box_lo[2] + (int)c2};
    int64_t lin = 0;
#pragma unroll
    for (int a = 0; a < B200NA_MAX_DIM; ++a)
      if (a < p.ax.ndim)
        lin = lin * p.ax.shape[a] + ((int64_t)x[a] * p.ax.dilation[a] + s.g[a]);
    row = (s.b * p.N + lin) * (kKeyRows ? p.Hq : p.Hkv) + head;
    cc = make_int4(x[0], x[1], x[2], kToken);
  } else if (j < n_all) {
    cc.w = kExtra;
  }
  c.row[slot] = row;
  c.c[slot] = cc;
}

// True when row r interacts with column c.
__device__ __forceinline__ bool pair_on(const Rows& s, int r, const int4& c, int nd) {
  if (c.w != kToken) return c.w == kExtra && s.row[r] >= 0;
  bool on = (unsigned)(c.x - s.lo[r][0]) < (unsigned)s.len[r][0];
  if (nd > 1) on = on && (unsigned)(c.y - s.lo[r][1]) < (unsigned)s.len[r][1];
  if (nd > 2) on = on && (unsigned)(c.z - s.lo[r][2]) < (unsigned)s.len[r][2];
  return on;
}

// `n` rows of D elements -> fp32 rows of DM + 4 floats in shared memory, zeros past D and for
// missing rows. The 4 floats of padding put rows 16 bytes apart in the banks, so that the eight
// rows a quarter-warp reads together cover all of them.
template <class T, int DM, bool kVec, int n>
__device__ __forceinline__ void load_rows(float* dst, const T* __restrict__ base,
                                          const int64_t* rows, int D) {
  constexpr int kChunks = DM / 4;
#pragma unroll 8
  for (int i = threadIdx.x; i < n * kChunks; i += kThreads) {
    const int r = i / kChunks, ch = i % kChunks;
    const int64_t row = rows[r];
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= 0) {
      const T* src = base + row * D + ch * 4;
      if (kVec) {
        if (ch * 4 < D) v = ldf4(src);
      } else {
        if (ch * 4 + 0 < D) v.x = ldf(src + 0);
        if (ch * 4 + 1 < D) v.y = ldf(src + 1);
        if (ch * 4 + 2 < D) v.z = ldf(src + 2);
        if (ch * 4 + 3 < D) v.w = ldf(src + 3);
      }
    }
    *reinterpret_cast<float4*>(dst + r * (DM + 4) + ch * 4) = v;
  }
}

// Keys and values of one step: token rows from k / v, then (slots from `n_tok - j0` on) extra
// tokens from tensors of their own.
template <class T, int DM, bool kVec>
__device__ __forceinline__ void load_key_values(const Params& p, const Rows& rows, const Cols& cols,
                                                int64_t j0, int64_t n_tok, int64_t n_all,
                                                float* k_sm, float* v_sm, const T* __restrict__ k,
                                                const T* __restrict__ v,
                                                const T* __restrict__ add_k,
                                                const T* __restrict__ add_v) {
  if (j0 < n_tok) {
    load_rows<T, DM, kVec, kCols>(k_sm, k, cols.row, p.D);
    load_rows<T, DM, kVec, kCols>(v_sm, v, cols.row, p.D);
  }
  if (p.n_extra > 0 && j0 + kCols > n_tok) {
    if (j0 < n_tok) __syncthreads();   // the slots below were just zeroed by other threads
    const int first = j0 < n_tok ? (int)(n_tok - j0) : 0;
    const int64_t e0 = rows.b * p.n_extra + j0 - n_tok;
    const int hk = rows.h / (p.Hq / p.Hkv);
    for (int i = threadIdx.x; i < (kCols - first) * DM; i += kThreads) {
      const int r = first + i / DM, c = i % DM;
      const bool on = j0 + r < n_all && c < p.D;
      const int64_t at = ((e0 + r) * p.Hkv + hk) * p.D + c;
      k_sm[r * (DM + 4) + c] = on ? ldf(add_k + at) : 0.f;
      v_sm[r * (DM + 4) + c] = on ? ldf(add_v + at) : 0.f;
    }
  }
}

// Thread layout of the products: 8 groups of 4 rows (`rg`) x 16 column lanes (`cl`); a warp holds
// two row groups, so everything about a row stays inside one warp.
// acc[r][i] += row (4 rg + r) . column (cl + 16 i), over the first `dp` (a multiple of 4) elements
template <int DM>
__device__ __forceinline__ void dot_tile(const float* rows, const float* cols, int rg, int cl, int dp,
                                         float (&acc)[4][4]) {
  const float* rp = rows + rg * 4 * (DM + 4);
  const float* cp = cols + cl * (DM + 4);
#pragma unroll 2
  for (int d = 0; d < dp; d += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = *reinterpret_cast<const float4*>(rp + r * (DM + 4) + d);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = *reinterpret_cast<const float4*>(cp + i * 16 * (DM + 4) + d);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[r][i] = fmaf(a[r].x, b[i].x, acc[r][i]);
        acc[r][i] = fmaf(a[r].y, b[i].y, acc[r][i]);
        acc[r][i] = fmaf(a[r].z, b[i].z, acc[r][i]);
        acc[r][i] = fmaf(a[r].w, b[i].w, acc[r][i]);
      }
  }
}
// Output columns of a thread: kW consecutive ones at kW cl + 16 kW m, kW = 4 (2 when DM = 32).
template <int DM>
struct OutCols {
  static constexpr int kW = DM >= 64 ? 4 : 2;
  static constexpr int kM = DM / (16 * kW);
  static constexpr int kPer = kW * kM;     // DM / 16
};
// acc[r][.] += sum_j w[4 rg + r][j] cols[j][.] over the first n4 (a multiple of 4) columns
template <int DM>
__device__ __forceinline__ void accumulate_tile(const float* w, const float* cols, int rg, int cl,
                                                int n4, float (&acc)[4][OutCols<DM>::kPer]) {
  using OC = OutCols<DM>;
  const float* wp = w + rg * 4 * kPStride;
#pragma unroll 2
  for (int j = 0; j < n4; j += 4) {
    float4 w4[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) w4[r] = *reinterpret_cast<const float4*>(wp + r * kPStride + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const float* cp = cols + (j + jj) * (DM + 4) + cl * OC::kW;
      float v[OC::kPer];
#pragma unroll
      for (int m = 0; m < OC::kM; ++m) {
        if constexpr (OC::kW == 4) {
          const float4 x = *reinterpret_cast<const float4*>(cp + m * 64);
          v[m * 4] = x.x; v[m * 4 + 1] = x.y; v[m * 4 + 2] = x.z; v[m * 4 + 3] = x.w;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(cp);
          v[0] = x.x; v[1] = x.y;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float f = jj == 0 ? w4[r].x : (jj == 1 ? w4[r].y : (jj == 2 ? w4[r].z : w4[r].w));
#pragma unroll
        for (int t = 0; t < OC::kPer; ++t) acc[r][t] = fmaf(f, v[t], acc[r][t]);
      }
    }
  }
}
// Non-finite columns. A column of the union box is multiplied with every row of the block, by zero where
// the pair does not interact, and 0 x NaN is NaN: a row would take over the NaN or infinity of a token
// outside its window. All that can reach a row that way makes its sums non-finite, so a block looks at
// its finished sums (one multiply-add each) and, if one is not finite, does the item again in a function
// that is not inlined (kAgain; a 32 x 32 map of 4 heads takes 22.5 us that way, as without the check, and
// 24.6 us with the second accumulation as a branch inside the loop). There the weights of pairs that do not interact are kNoWeight, which
// no interacting pair has, and are skipped.
constexpr unsigned kNoWeight = 0x80000000u;   // -0
__device__ __forceinline__ float weight_if(bool on, float w) {
  return on ? w + 0.f : __uint_as_float(kNoWeight);   // -0 + 0 = +0
}
template <int DM>
__device__ __forceinline__ void accumulate_interacting(const float* w, const float* cols, int rg, int cl,
                                                       int n4, float (&acc)[4][OutCols<DM>::kPer]) {
  using OC = OutCols<DM>;
#pragma unroll 1
  for (int j = 0; j < n4; ++j) {
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float f = w[(rg * 4 + r) * kPStride + j];
      if (__float_as_uint(f) == kNoWeight) continue;
#pragma unroll
      for (int t = 0; t < OC::kPer; ++t)
        acc[r][t] = fmaf(f, cols[j * (DM + 4) + (t / OC::kW) * 16 * OC::kW + cl * OC::kW + t % OC::kW],
                         acc[r][t]);
    }
  }
}
template <int kN>
__device__ __forceinline__ bool any_non_finite(const float (&acc)[4][kN]) {
  float t = 0.f;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int i = 0; i < kN; ++i) t = fmaf(acc[r][i], 0.f, t);
  return t != 0.f;   // NaN
}
template <class T, int DM>
__device__ __forceinline__ void store_row(T* dst, const float (&acc)[OutCols<DM>::kPer], float mul,
                                          int cl, int D) {
  using OC = OutCols<DM>;
#pragma unroll
  for (int t = 0; t < OC::kPer; ++t) {
    const int col = (t / OC::kW) * 16 * OC::kW + cl * OC::kW + t % OC::kW;
    if (col < D) stf(dst + col, acc[t] * mul);
  }
}
// reductions over the 16 lanes that share a row
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- host ------------------------------------------------------------------------------------------

// Row tile shape and item count. The shape is the factorisation of 32 that visits the fewest column
// steps (row tiles times 64-column steps over the union box); ties go to the tile that is longest
// along the last axis.
inline void plan_rows(Params& p) {
  p.T[0] = kRows; p.T[1] = p.T[2] = 1;
  if (!p.dense && !p.extra_rows && p.ax.ndim > 1) {
    double best = 1e300;
    for (int e0 = 5; e0 >= 0; --e0)
      for (int e1 = 5 - e0; e1 >= 0; --e1) {
        const int e2 = 5 - e0 - e1;
        if (p.ax.ndim == 2 && e2 != 0) continue;
        const int t[B200NA_MAX_DIM] = {1 << e0, 1 << e1, 1 << e2};
        double tiles = 1., cols = 1.;
        for (int a = 0; a < p.ax.ndim; ++a) {
          const int L = (p.ax.shape[a] + p.ax.dilation[a] - 1) / p.ax.dilation[a];
          const int s = p.ax.stride[a];
          tiles *= (L + t[a] - 1) / t[a];
          const int leaders = (t[a] + s - 1) / s;   // stride groups an aligned tile spans
          cols *= imin(L, p.ax.kernel[a] + (leaders - 1) * s);
        }
        const double steps = cols < kCols ? 1. : cols / kCols;
        if (tiles * steps <= best) {
          best = tiles * steps;
          for (int a = 0; a < B200NA_MAX_DIM; ++a) p.T[a] = t[a];
        }
      }
  }
  for (int a = 0; a < B200NA_MAX_DIM; ++a) {
    int64_t ext = 1;
    if (p.extra_rows) ext = a == 0 ? p.n_extra : 1;
    else if (p.dense) ext = a == 0 ? p.Nq : 1;
    else if (a < p.ax.ndim) ext = (p.ax.shape[a] + p.ax.dilation[a] - 1) / p.ax.dilation[a];
    p.R[a] = (int)((ext + p.T[a] - 1) / p.T[a]);
  }
  p.n_items = (int64_t)p.R[0] * p.R[1] * p.R[2] * p.row_heads * p.B * p.G;
}

// 4-element vector access: every row starts on a multiple of 4 elements.
inline bool vectorised(int D, size_t elem_bytes, uintptr_t all_pointers) {
  return D % 4 == 0 && all_pointers % (4 * elem_bytes) == 0;
}

// Launches `fn` with one block per item and opt-in shared memory (set once per kernel and device).
int launch(const void* fn, int64_t items, int smem_bytes, void** args, cudaStream_t stream);

}  // namespace simt
}  // namespace b200na
