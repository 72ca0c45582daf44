// Native front of the operators for eager PyTorch calls: argument parsing, checks, tile choice,
// allocation, launch and autograd without Python in between.
//
// Why: the kernels of a small map take 10-20 us, while a call through torch.library.custom_op, the
// Python checks and ctypes took 90-160 us of host time (forward alone; training twice that). Here
// a forward is one C call: parse, check, two allocations, tensor maps, launch. The Python front
// (functional.py) keeps the registered operators for torch.compile, fake tensors, function
// transforms and every call this file does not take: a function returns None for those - including
// every invalid argument, so that messages and exception types stay in one place.
//
// Threads and streams: nothing is kept between calls but the tile-shape plans (bounded, under a
// mutex); launches go to the caller's current stream. Double backward is refused.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <dlfcn.h>

#include <ATen/ATen.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <pybind11/pybind11.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <optional>
#include <utility>
#include <vector>

#include "../../include/natten_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr int kMaxDim = 3;

// ---- the C library (the one the Python package loaded) -----------------------------------------
#define B200NA_FUNCTIONS(X)                                                                  \
  X(na_forward_view) X(na_forward_simt) X(fmha_forward) X(fmha_splits) X(fmha_forward_split)  \
  X(na_backward_view) X(na_backward_simt)                                                     \
  X(column_sum) X(column_sum_scratch) X(strerror)
struct Lib {
#define X(name) decltype(&b200na_##name) name = nullptr;
  B200NA_FUNCTIONS(X)
#undef X
} lib;
std::atomic<long long> launches{0};

void check(int code, const char* where) {
  TORCH_CHECK(code == B200NA_OK, where, " failed with code ", code, ": ", lib.strerror(code));
}

// ---- window arithmetic and tile shapes -----------------------------------------------------------
// (same integer semantics as the kernels; reference csrc/include/natten/cuda/reference/
// mask.hpp:47-89, 220-225)
int window_start(int i, int k, int s, int L, bool causal) {
  const int wl = k / 2, wr = k / 2 + (k % 2 - 1);
  if (causal) {
    const int lead = std::min((i / s) * s + s - 1, L - 1);
    return std::max(lead - wl - wr, 0);
  }
  const int lead = std::min((i / s) * s + s / 2, L - 1);
  return std::max(lead - wl, 0) + (lead + wr >= L ? L - wr - lead - 1 : 0);
}
int window_end(int i, int start, int k, int L, bool causal) {
  return causal ? std::min(i + 1, L) : start + k;
}
int ceil_div(int a, int b) { return (a + b - 1) / b; }

struct Problem {
  int nd = 0;
  std::array<int, kMaxDim> shape{1, 1, 1}, kernel{1, 1, 1}, stride{1, 1, 1}, dilation{1, 1, 1},
      causal{0, 0, 0};
  bool operator<(const Problem& o) const {
    return std::tie(nd, shape, kernel, stride, dilation, causal) <
           std::tie(o.nd, o.shape, o.kernel, o.stride, o.dilation, o.causal);
  }
};
struct Tiles {
  std::array<int, kMaxDim> q{1, 1, 1}, kv{1, 1, 1};
};

constexpr int kQTile = 256, kHalfQTile = 128, kKVTile = 128;
// A 128-token query tile pays with twice the key/value tile loads per query row and a shallower
// load ring: its tile count is charged this factor.
constexpr double kSmallQTilePenalty = 1.15;
constexpr int kMaxBox = 256, kMaxElementStride = 8;   // limits of a tensor-map box

// KV tiles visited along one axis, summed over its query tiles (largest dilation group). `aligned`:
// the walk starts at the first key the tile's queries attend, otherwise on a grid from 0.
long long axis_tile_cost(const Problem& p, int a, int tq, int tkv, bool aligned) {
  const int L = ceil_div(p.shape[a], p.dilation[a]), k = p.kernel[a], s = p.stride[a];
  const bool c = p.causal[a];
  long long total = 0;
  for (int lo = 0; lo < L; lo += tq) {
    const int hi = lo + tq - 1;
    const int st = window_start(lo, k, s, L, c);
    const int en = window_end(hi, window_start(hi, k, s, L, c), k, L, c);
    total += aligned ? ceil_div(en - st, tkv) : ceil_div(en, tkv) - st / tkv;
  }
  return total;
}
// Query tiles visited along one axis, summed over its key tiles, by the pass whose stationary tile
// holds keys: from the first query that attends one of the tile's keys to the last.
long long axis_inverse_tile_cost(const std::vector<int>& starts, const std::vector<int>& ends, int tq,
                                 int tkv) {
  const int L = (int)starts.size();
  long long total = 0;
  for (int lo = 0; lo < L; lo += tkv) {
    const int hi = std::min(lo + tkv, L) - 1;
    const long long first = std::upper_bound(ends.begin(), ends.end(), lo) - ends.begin();
    const long long last = std::upper_bound(starts.begin(), starts.end(), hi) - starts.begin();
    total += std::max(1ll, (last - first + tq - 1) / tq);
  }
  return total;
}

std::vector<std::array<int, kMaxDim>> compositions(int log2_total, int n) {
  std::vector<std::array<int, kMaxDim>> out;
  for (int e0 = 0; e0 <= log2_total; ++e0)
    for (int e1 = 0; e0 + e1 <= log2_total; ++e1) {
      const int e2 = log2_total - e0 - e1;
      if ((n < 2 && (e1 || e2)) || (n < 3 && e2)) continue;
      out.push_back({1 << e0, 1 << e1, 1 << e2});
    }
  return out;
}
bool box_fits(const std::array<int, kMaxDim>& tile, const Problem& p) {
  for (int a = 0; a < p.nd; ++a)
    if (p.dilation[a] > kMaxElementStride || tile[a] * p.dilation[a] > kMaxBox) return false;
  return true;
}
// Whether the forward kernel can read the caller's layout with these tiles: a 256-token query tile is
// fetched as two halves split along its last non-unit axis.
bool direct_supported(std::array<int, kMaxDim> q, const std::array<int, kMaxDim>& kv,
                      const Problem& p) {
  int total = 1, split = 0;
  for (int a = 0; a < p.nd; ++a) {
    total *= q[a];
    if (q[a] > 1) split = a;
  }
  if (total > kHalfQTile) {
    if (q[split] % 2) return false;
    q[split] /= 2;
  }
  return box_fits(q, p) && box_fits(kv, p);
}

int log2i(int x) {
  int e = 0;
  while ((1 << e) < x) ++e;
  return e;
}

// (q tile, kv tile) - 256 or 128 query tokens, 128 key/value tokens - that minimise the tile products
// the forward kernel computes; ties to tiles that are long along the last (contiguous) axis.
Tiles choose_forward(const Problem& p) {
  Tiles t;
  if (p.nd == 1) {
    t.q[0] = kQTile;
    t.kv[0] = kKVTile;
    return t;
  }
  double cost[kMaxDim][9][8][2];
  for (int a = 0; a < p.nd; ++a)
    for (int eq = 0; eq < 9; ++eq)
      for (int ek = 0; ek < 8; ++ek)
        for (int al = 0; al < 2; ++al)
          cost[a][eq][ek][al] = (double)axis_tile_cost(p, a, 1 << eq, 1 << ek, al);
  std::array<double, 3> best{1e300, 0, 0};
  const auto kvs = compositions(7, p.nd);
  for (int half = 0; half < 2; ++half)
    for (const auto& q : compositions(half ? 7 : 8, p.nd))
      for (const auto& kv : kvs) {
        const int al = direct_supported(q, kv, p);
        double c = half ? kSmallQTilePenalty : 2.0;
        for (int a = 0; a < p.nd; ++a) c *= cost[a][log2i(q[a])][log2i(kv[a])][al];
        const std::array<double, 3> key{c, -(double)q[p.nd - 1], -(double)kv[p.nd - 1]};
        if (key < best) {
          best = key;
          t.q = q;
          t.kv = kv;
        }
      }
  return t;
}
// 128-token tiles for the two backward passes: key/value tiles per query tile (dQ) plus query tiles
// per key/value tile (dK, dV). No pair that fits a box: unusable tiles (the caller then takes the
// CUDA-core kernels).
Tiles choose_backward(const Problem& p) {
  Tiles t;
  t.q[0] = t.kv[0] = 128;
  if (p.nd == 1) return t;
  double cost[kMaxDim][8][8][2];
  for (int a = 0; a < p.nd; ++a) {
    const int L = ceil_div(p.shape[a], p.dilation[a]);
    std::vector<int> starts(L), ends(L);
    for (int i = 0; i < L; ++i) {
      starts[i] = window_start(i, p.kernel[a], p.stride[a], L, p.causal[a]);
      ends[i] = window_end(i, starts[i], p.kernel[a], L, p.causal[a]);
    }
    for (int eq = 0; eq < 8; ++eq)
      for (int ek = 0; ek < 8; ++ek) {
        cost[a][eq][ek][0] = (double)axis_tile_cost(p, a, 1 << eq, 1 << ek, true);
        cost[a][eq][ek][1] = (double)axis_inverse_tile_cost(starts, ends, 1 << eq, 1 << ek);
      }
  }
  std::array<double, 3> best{1e300, 0, 0};
  const auto tiles = compositions(7, p.nd);
  for (const auto& q : tiles) {
    if (!box_fits(q, p)) continue;
    for (const auto& kv : tiles) {
      if (!box_fits(kv, p)) continue;
      double c0 = 1, c1 = 1;
      for (int a = 0; a < p.nd; ++a) {
        c0 *= cost[a][log2i(q[a])][log2i(kv[a])][0];
        c1 *= cost[a][log2i(q[a])][log2i(kv[a])][1];
      }
      const std::array<double, 3> key{c0 + c1, -(double)q[p.nd - 1], -(double)kv[p.nd - 1]};
      if (key < best) {
        best = key;
        t.q = q;
        t.kv = kv;
      }
    }
  }
  return t;
}
// ---- tiles of any size up to the kernels' (the entries for views) -------------------------------------
// A tile need not hold exactly 128 (256) tokens, nor powers of two of them: 15 rows are one tile of 15.
// The rows that remain are zeros in shared memory and masked. Tiles computed against powers of two:
// 14 x 21 x 22 with 14 x 21 x 9 windows -49 %, 10 x 49 x 19 with 8 x 6 x 5 -32 %, 29 x 21 with 11 x 8
// -19 %; none where extents and windows are powers of two already.

// Column tokens a stationary tile meets along an axis, and of these [lo, hi), counted from the first,
// inside the window of every row; `count` tiles of the axis are alike.
struct Run {
  int span, lo, hi;
  long long count;
};
using Runs = std::vector<Run>;
void add_run(Runs& r, int span, int lo, int hi) {
  for (auto it = r.rbegin(); it != r.rend() && it - r.rbegin() < 4; ++it)
    if (it->span == span && it->lo == lo && it->hi == hi) {
      ++it->count;
      return;
    }
  r.push_back({span, lo, hi, 1});
}
// Windows of one axis (the largest dilation group): queries attend [start, end).
struct AxisWindows {
  int L = 0;
  std::vector<int> start, end;
};
AxisWindows axis_windows(const Problem& p, int a) {
  AxisWindows w;
  w.L = ceil_div(p.shape[a], p.dilation[a]);
  w.start.resize(w.L);
  w.end.resize(w.L);
  for (int i = 0; i < w.L; ++i) {
    w.start[i] = window_start(i, p.kernel[a], p.stride[a], w.L, p.causal[a]);
    w.end[i] = window_end(i, w.start[i], p.kernel[a], w.L, p.causal[a]);
  }
  return w;
}
Runs query_runs(const AxisWindows& w, int tile) {
  Runs r;
  for (int lo = 0; lo < w.L; lo += tile) {
    const int hi = std::min(lo + tile, w.L) - 1;
    add_run(r, w.end[hi] - w.start[lo], w.start[hi] - w.start[lo], w.end[lo] - w.start[lo]);
  }
  return r;
}
Runs key_runs(const AxisWindows& w, int tile) {
  Runs r;
  const auto first = [&](int j) { return (int)(std::upper_bound(w.end.begin(), w.end.end(), j) - w.end.begin()); };
  const auto last = [&](int j) { return (int)(std::upper_bound(w.start.begin(), w.start.end(), j) - w.start.begin()); };
  for (int lo = 0; lo < w.L; lo += tile) {
    const int hi = std::min(lo + tile, w.L) - 1, f = first(lo);
    add_run(r, last(hi) - f, first(hi) - f, last(lo) - f);
  }
  return r;
}
// column tiles of all the axis' stationary tiles, and how many of these need no mask
std::array<double, 2> tiles_met(const Runs& runs, int tile) {
  long long all = 0, inside = 0;
  for (const Run& r : runs) {
    all += r.count * std::max(1, ceil_div(r.span, tile));
    inside += r.count * std::max(0, std::max(r.hi, 0) / tile - ceil_div(r.lo, tile));
  }
  return {(double)all, (double)inside};
}
// Sizes worth trying for a length: those that cut it into equal parts, and the powers of two.
std::vector<int> part_sizes(int length, int most) {
  std::vector<int> out;
  for (int n = 1; n <= length; ++n) {
    const int t = ceil_div(length, n);
    if (t <= most && (out.empty() || out.back() != t)) out.push_back(t);
  }
  for (int t = 1; t <= most && t < 2 * length; t *= 2) out.push_back(t);
  std::sort(out.begin(), out.end());
  out.erase(std::unique(out.begin(), out.end()), out.end());
  return out;
}
// Tiles of `nd` axes with sizes out of `sizes`, at most `most` tokens: the last axis takes the largest
// size that fits the others.
void tiles_within(const std::vector<int>* const (&sizes)[kMaxDim], int nd, int most,
                  std::vector<std::array<int, kMaxDim>>& out) {
  const std::vector<int> one{1};
  const auto& s0 = nd >= 2 ? *sizes[0] : one;
  const auto& s1 = nd >= 3 ? *sizes[1] : one;
  for (int a : s0)
    for (int b : s1) {
      if (a * b > most) break;
      const auto& s = *sizes[nd - 1];
      const auto it = std::upper_bound(s.begin(), s.end(), most / (a * b));
      if (it == s.begin()) continue;
      std::array<int, kMaxDim> t{1, 1, 1};
      t[0] = a;
      if (nd >= 3) t[1] = b;
      t[nd - 1] = *std::prev(it);
      out.push_back(t);
    }
}
int tokens_of(const std::array<int, kMaxDim>& t) { return t[0] * t[1] * t[2]; }

// An item's own cost (descriptor, first loads, epilogue) in tiles, and what a tile without a mask
// costs of one with: from the kernels' cycle counters (3650 against 4800 cycles a tile, about 5000 an
// item; the backward masks half as many values).
constexpr double kItemTiles = 1.3, kForwardInside = 0.9, kBackwardInside = 0.9;
// A column tile of fewer than 128 tokens is charged more than its share of the tiles: at 9 % fewer tiles
// (56 x 56, 7 x 7) and 5 % fewer (128 x 128, 13 x 13, dilation 2) the forward came out 4 % and 5 % slower
// than with full ones, where tiles drop by 20 % and more 18 to 27 % faster.
constexpr double kRaggedForward = 1.1, kRaggedBackward = 1.06;
// The plan of powers of two stays unless another is estimated this much cheaper: the estimate is good to
// some percent (15 x 30 x 52, 7 x 15 x 15: estimated 7 % cheaper, the training step 2 % slower).
constexpr double kWorthwhile = 0.9;

// Tile pair of least cost. `exact_kv`: key/value tiles of exactly 128 tokens (extra tokens).
bool choose_view(const Problem& p, bool backward, bool exact_kv, Tiles* best) {
  AxisWindows win[kMaxDim];
  std::vector<int> sizes[kMaxDim];
  const std::vector<int>* const size_lists[kMaxDim] = {&sizes[0], &sizes[1], &sizes[2]};
  for (int a = 0; a < p.nd; ++a) win[a] = axis_windows(p, a);
  std::vector<std::array<int, kMaxDim>> qs;
  for (int most = 128; most <= (backward ? 128 : 256); most *= 2) {
    for (int a = 0; a < p.nd; ++a) sizes[a] = part_sizes(win[a].L, most);
    tiles_within(size_lists, p.nd, most, qs);
  }
  // worked out as they are asked for: runs by rows, tiles met by rows and columns
  constexpr int kRows = 257, kCols = 129;
  std::vector<Runs> runs[2][kMaxDim];
  std::vector<std::array<double, 2>> met[2][kMaxDim];
  for (int pass = 0; pass < (backward ? 2 : 1); ++pass)
    for (int a = 0; a < p.nd; ++a) {
      runs[pass][a].resize(kRows);
      met[pass][a].assign(kRows * kCols, {-1, 0});
    }
  const auto runs_of = [&](int pass, int a, int rows) -> const Runs& {
    Runs& r = runs[pass][a][rows];
    if (r.empty()) r = pass ? key_runs(win[a], rows) : query_runs(win[a], rows);
    return r;
  };
  const auto column_tiles = [&](int pass, int a, int rows, int cols) -> const std::array<double, 2>& {
    auto& m = met[pass][a][rows * kCols + cols];
    if (m[0] < 0) m = tiles_met(runs_of(pass, a, rows), cols);
    return m;
  };
  std::map<int, std::vector<int>> cuts[kMaxDim];   // key/value sizes worth trying, by query rows
  const auto cost = [&](const std::array<int, kMaxDim>& q, const std::array<int, kMaxDim>& kv) {
    const int nq = tokens_of(q);
    const bool full = tokens_of(kv) == kKVTile;
    double all = 1, in = 1, q_items = 1;
    for (int a = 0; a < p.nd; ++a) {
      const auto& m = column_tiles(0, a, q[a], kv[a]);
      q_items *= ceil_div(win[a].L, q[a]);
      all *= m[0];
      in *= m[1];
    }
    double c = all + kItemTiles * q_items;
    if (full) c -= (1 - (backward ? kBackwardInside : kForwardInside)) * in;
    else c *= backward ? kRaggedBackward : kRaggedForward;
    if (!backward) return c * (nq <= kHalfQTile ? kSmallQTilePenalty : 2.0);
    double k_items = 1;
    all = in = 1;
    for (int a = 0; a < p.nd; ++a) {
      k_items *= ceil_div(win[a].L, kv[a]);
      const auto& m = column_tiles(1, a, kv[a], q[a]);
      all *= m[0];
      in *= m[1];
    }
    return c + (all + kItemTiles * k_items - (1 - kBackwardInside) * in) *
                   (nq == kHalfQTile ? 1.0 : kRaggedBackward);
  };
  double least = 1e300;
  std::vector<std::array<int, kMaxDim>> kvs;
  for (const auto& q : qs) {
    if (backward ? !box_fits(q, p) : !direct_supported(q, {1, 1, 1}, p)) continue;
    kvs.clear();
    const std::vector<int>* cut[kMaxDim] = {};
    for (int a = 0; a < p.nd; ++a) {
      std::vector<int>& c = cuts[a][q[a]];
      if (c.empty()) {
        int last = 0;
        for (const Run& r : runs_of(0, a, q[a])) {
          const int span = std::min(r.span, 128);
          if (span == last) continue;
          last = span;
          const std::vector<int> s = part_sizes(span, 128);
          c.insert(c.end(), s.begin(), s.end());
        }
        std::sort(c.begin(), c.end());
        c.erase(std::unique(c.begin(), c.end()), c.end());
      }
      cut[a] = &c;
    }
    if (exact_kv) kvs = compositions(7, p.nd);
    else tiles_within(cut, p.nd, 128, kvs);
    for (const auto& kv : kvs) {
      if (!box_fits(kv, p)) continue;
      // ties go to full tiles, then to such as are long along the last (contiguous) axis
      const double c = cost(q, kv) * (1 - 1e-9 * ((tokens_of(kv) == kKVTile ? 512 : 0) + q[p.nd - 1] +
                                                  kv[p.nd - 1] / 256.0));
      if (c < least) {
        least = c;
        best->q = q;
        best->kv = kv;
      }
    }
  }
  const Tiles even = backward ? choose_backward(p) : choose_forward(p);
  if ((backward ? box_fits(even.q, p) && box_fits(even.kv, p) : direct_supported(even.q, even.kv, p)) &&
      cost(even.q, even.kv) * kWorthwhile <= least)
    *best = even;
  return least < 1e300;
}

// Plans are kept per problem (at most kMaxPlans, then the store starts over).
Tiles plan(const Problem& p, bool backward, bool extra) {
  if (p.nd == 1) return backward ? choose_backward(p) : choose_forward(p);
  constexpr size_t kMaxPlans = 1024;
  static std::mutex mu;
  static std::map<Problem, Tiles> stores[2][2];
  auto& store = stores[extra];
  {
    std::lock_guard<std::mutex> lk(mu);
    auto it = store[backward].find(p);
    if (it != store[backward].end()) return it->second;
  }
  Tiles t;
  // no pair that fits a tensor-map box: tiles the caller then finds unusable
  if (!choose_view(p, backward, extra, &t)) t = backward ? choose_backward(p) : choose_forward(p);
  std::lock_guard<std::mutex> lk(mu);
  if (store[backward].size() >= kMaxPlans) store[backward].clear();
  store[backward][p] = t;
  return t;
}

// ---- operands -----------------------------------------------------------------------------------

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return B200NA_F32;
    case at::kHalf: return B200NA_F16;
    case at::kBFloat16: return B200NA_BF16;
    case at::kFloat8_e4m3fn: return B200NA_E4M3;
    case at::kFloat8_e5m2: return B200NA_E5M2;
    default: return -1;
  }
}
bool is_16bit(int dt) { return dt == B200NA_F16 || dt == B200NA_BF16; }
bool is_8bit(int dt) { return dt == B200NA_E4M3 || dt == B200NA_E5M2; }
// head dims the tensor-core kernels read as they lie
bool reads_natively(int dt, int D) {
  if (is_16bit(dt)) return D >= 8 && D <= 128 && D % 8 == 0;
  return is_8bit(dt) && D >= 16 && D <= 128 && D % 16 == 0;
}

// Elements between consecutive tokens of a heads-last tensor whose tokens (batch entries included)
// are evenly spaced and whose [H, D] block is contiguous; -1 when it is not of that form or not
// aligned for a tensor map. The stride of an axis of one entry means nothing and is not looked at:
// [B, 1, N, D] transposed to [B, N, 1, D] has a head stride of N D.
long long token_stride(const Tensor& t) {
  const int n = (int)t.dim();
  const int64_t H = t.size(n - 2), D = t.size(n - 1);
  if ((D != 1 && t.stride(n - 1) != 1) || (H != 1 && t.stride(n - 2) != D)) return -1;
  int64_t ts = H * D, expected = -1;
  for (int i = n - 3; i >= 0; --i) {
    if (t.size(i) == 1) continue;
    if (expected < 0) ts = expected = t.stride(i);   // innermost axis of more than one token
    if (t.stride(i) != expected) return -1;
    expected *= t.size(i);
  }
  if (ts < H * D || (ts * t.element_size()) % 16 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16)
    return -1;
  return ts;
}
// a token-strided tensor (a contiguous one when it is not) and its stride, 0 = contiguous
struct View {
  Tensor t;
  long long ts;
};
View as_view(const Tensor& t) {
  const long long ts = token_stride(t);
  if (ts >= 0) return {t, ts};
  return {t.contiguous(), 0};
}

// A contiguous tensor on a 16-byte boundary, as the tensor-core backward and the column sums read an
// output gradient. A piece of a flat buffer (split, cat's backward) is contiguous wherever it starts.
Tensor aligned(const Tensor& t) {
  Tensor c = t.contiguous();
  if (reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 != 0) c = c.clone(at::MemoryFormat::Contiguous);
  return c;
}

// tokens of a batch entry of a heads-last tensor (its sizes' product may need 64 bits: callers check it)
int64_t token_count(const Tensor& t) {
  int64_t n = 1;
  for (int64_t i = 1; i < t.dim() - 2; ++i) n *= t.size(i);
  return n;
}

struct Sizes {
  int B, Hq, Hkv, D, dt;
};
b200na_stream_t stream_of(const Tensor& t) {
  return (b200na_stream_t)c10::cuda::getCurrentCUDAStream(t.get_device()).stream();
}
// launches of a call: a folded 1-D dilation needs one per kind of group
int parts_of(const Problem& p) {
  const int d = p.dilation[0];
  return p.nd == 1 && d > 2 && p.shape[0] % d ? 2 : 1;
}

struct Pointers {
  const void *q, *k, *v;
  long long q_ts, k_ts, v_ts;
  const void *ak, *av;
  int n_extra;
};

// Kernel choice for a forward call. kNone: not taken here.
enum class Path { kNone, kTensorCore, kCudaCore };
Path forward_path(const Problem& p, const Sizes& z, bool extra, Tiles* tiles) {
  bool tensor_core = reads_natively(z.dt, z.D);
  if (p.nd == 3 && !is_8bit(z.dt))
    for (int a = 0; a < 3; ++a)
      if (p.shape[a] >= 65536) tensor_core = false;   // window bounds are kept in 16 bits there
  if (!tensor_core) {
    // 16-bit head dims below 128 that are not multiples of 8 are zero-padded first
    if (is_8bit(z.dt) || z.D > 256 || (is_16bit(z.dt) && z.D < 128)) return Path::kNone;
    return Path::kCudaCore;
  }
  if (p.nd == 3 && z.B > 1 && z.D != 128 && (is_8bit(z.dt) || z.D != 64)) return Path::kNone;
  *tiles = plan(p, false, extra);
  if (p.nd > 1 && !direct_supported(tiles->q, tiles->kv, p)) return Path::kNone;
  return Path::kTensorCore;
}
int run_forward(const Problem& p, const Sizes& z, float scale, Path path, const Tiles& t,
                const Pointers& a, void* out, float* lse, b200na_stream_t stream) {
  int rc;
  if (path == Path::kTensorCore) {
    rc = lib.na_forward_view(a.q, a.k, a.v, a.ak, a.av, a.n_extra, out, lse, p.nd, p.shape.data(),
                             p.kernel.data(), p.stride.data(), p.dilation.data(), p.causal.data(),
                             t.q.data(), t.kv.data(), z.B, z.Hq, z.Hkv, z.D, z.dt, scale, a.q_ts,
                             a.k_ts, a.v_ts, stream);
    if (rc == B200NA_OK) launches += parts_of(p);
  } else {
    rc = lib.na_forward_simt(a.q, a.k, a.v, out, lse, p.nd, p.shape.data(), p.kernel.data(),
                             p.stride.data(), p.dilation.data(), p.causal.data(), z.B, z.Hq, z.Hkv,
                             z.D, z.dt, scale, a.ak, a.av, a.n_extra, stream);
    if (rc == B200NA_OK) ++launches;
  }
  return rc;
}

// ---- backward -------------------------------------------------------------------------------------

struct GradPointers {
  void *dq, *dk, *dv;
  long long dq_ts, dk_ts, dv_ts;   // tensor-core path only; the CUDA-core path needs 0 (contiguous)
  void *dak, *dav;
};
// Gradients whose P and dS keep more bits than the operands have: dense attention (a window over all of
// one axis) and 1-D dilation above 2.
bool exact_gradients(const Problem& p, bool extra) {
  return p.nd == 1 && (p.dilation[0] > 2 || (!extra && p.kernel[0] == p.shape[0]));
}
// Sums of more terms than this have an error of their own beside fp16's results on the tensor cores, whose
// accumulators round towards zero: 2 % of it at 16384 terms, 25 to 45 % at 65536.
constexpr int kMostExactTermsF16 = 4096;
bool backward_on_tensor_cores(const Problem& p, const Sizes& z, bool extra, Tiles* t) {
  if (!is_16bit(z.dt) || !reads_natively(z.dt, z.D)) return false;
  if (z.dt == B200NA_F16 && exact_gradients(p, extra) &&
      (extra ? p.shape[0] : p.kernel[0]) > kMostExactTermsF16)
    return false;
  if (p.nd == 3 && z.B > 1 && z.D != 64 && z.D != 128) return false;
  *t = plan(p, true, extra);
  return p.nd == 1 || (box_fits(t->q, p) && box_fits(t->kv, p));
}
void run_backward(const Problem& p, const Sizes& z, float scale, bool tensor_core, const Tiles& t,
                  const Pointers& a, const void* out, const void* d_out, const float* lse,
                  const GradPointers& g, float* delta, b200na_stream_t stream) {
  if (tensor_core) {
    check(lib.na_backward_view(a.q, a.k, a.v, out, d_out, lse, a.ak, a.av, a.n_extra, g.dq, g.dk, g.dv,
                               g.dak, g.dav, delta, p.nd, p.shape.data(), p.kernel.data(),
                               p.stride.data(), p.dilation.data(), p.causal.data(), t.q.data(),
                               t.kv.data(), z.B, z.Hq, z.Hkv, z.D, z.dt, scale, a.q_ts, a.k_ts, a.v_ts,
                               g.dq_ts, g.dk_ts, g.dv_ts, stream),
          "b200na_na_backward_view");
    launches += 1 + 2 * parts_of(p) + (a.n_extra ? 1 : 0);
    if (exact_gradients(p, a.n_extra))   // row norms; a look for non-finite rows where there are masks
      launches += (z.dt == B200NA_F16 ? 1 : 0) + (p.dilation[0] > 2 || p.causal[0] ? 2 : 0);
  } else {
    check(lib.na_backward_simt(a.q, a.k, a.v, out, d_out, lse, a.ak, a.av, a.n_extra, g.dq, g.dk, g.dv,
                               g.dak, g.dav, delta, p.nd, p.shape.data(), p.kernel.data(),
                               p.stride.data(), p.dilation.data(), p.causal.data(), z.B, z.Hq, z.Hkv,
                               z.D, z.dt, scale, stream),
          "b200na_na_backward_simt");
    launches += a.n_extra ? 3 : 2;
  }
}

// A backward whose results are differentiated again has no formula: with grad mode on (create_graph)
// they leave through this node, whose own backward refuses.
struct NoDoubleBackward : torch::autograd::Function<NoDoubleBackward> {
  static variable_list forward(AutogradContext*, at::TensorList in) {
    variable_list out;
    for (const auto& g : in) out.push_back(g.view_as(g));
    return out;
  }
  static variable_list backward(AutogradContext*, variable_list) {
    TORCH_CHECK(false, "natten_b200: the gradients of neighborhood attention cannot be differentiated "
                       "again (no double backward).");
  }
};
variable_list seal(variable_list grads) {
  if (!c10::GradMode::is_enabled()) return grads;
  variable_list on;
  for (auto& g : grads)
    if (g.defined()) on.push_back(g.requires_grad_());
  on = NoDoubleBackward::apply(at::TensorList(on));
  size_t i = 0;
  for (auto& g : grads)
    if (g.defined()) g = on[i++];
  return grads;
}

struct Call {
  Problem p;
  Sizes z{};
  float scale = 0.f;
  bool dense = false;      // dense attention (its backward: a window of the whole sequence)
  Path path = Path::kNone;
  Tiles tiles;
};

// (out, lse) of one forward; lse is undefined when it is not wanted. status != 0: nothing usable.
struct Forward {
  Tensor out, lse;
  int status;
};
Forward forward_now(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ak,
                    const Tensor& av, bool want_lse) {
  Forward f;
  c10::cuda::CUDAGuard guard(q.device());
  f.out = at::empty(q.sizes(), q.options());
  if (want_lse) f.lse = at::empty(q.sizes().slice(0, q.dim() - 1), q.options().dtype(at::kFloat));
  float* lse = want_lse ? f.lse.data_ptr<float>() : nullptr;
  b200na_stream_t stream = stream_of(q);
  if (c.dense) {
    const Tensor qc = q.contiguous(), kc = k.contiguous(), vc = v.contiguous();
    const int nq = (int)token_count(q), nk = (int)token_count(k);
    const int splits =
        c.scale > 0.f ? lib.fmha_splits(c.z.B, nq, nk, c.z.Hq, c.z.D, c.z.dt, c.p.causal[0]) : 1;
    if (splits > 1) {
      const Tensor scratch = at::empty({(int64_t)splits * c.z.B * nq * c.z.Hq * (c.z.D + 1)},
                                       q.options().dtype(at::kFloat));
      f.status = lib.fmha_forward_split(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), f.out.data_ptr(),
                                        lse, c.z.B, nq, nk, c.z.Hq, c.z.Hkv, c.z.D, c.z.dt, c.scale,
                                        scratch.data_ptr<float>(), stream);
      if (f.status == B200NA_OK) launches += 2;
      return f;
    }
    f.status = lib.fmha_forward(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), f.out.data_ptr(), lse,
                                c.z.B, nq, nk, c.z.Hq, c.z.Hkv, c.z.D, c.z.dt, c.scale,
                                c.p.causal[0], stream);
    if (f.status == B200NA_OK) ++launches;
    return f;
  }
  View qv, kv, vv;
  if (c.path == Path::kTensorCore) {
    qv = as_view(q); kv = as_view(k); vv = as_view(v);
  } else {
    qv = {q.contiguous(), 0}; kv = {k.contiguous(), 0}; vv = {v.contiguous(), 0};
  }
  Tensor akc, avc;
  if (ak.defined()) { akc = ak.contiguous(); avc = av.contiguous(); }
  const Pointers a{qv.t.data_ptr(), kv.t.data_ptr(), vv.t.data_ptr(), qv.ts, kv.ts, vv.ts,
                   ak.defined() ? akc.data_ptr() : nullptr, ak.defined() ? avc.data_ptr() : nullptr,
                   ak.defined() ? (int)ak.size(1) : 0};
  f.status = run_forward(c.p, c.z, c.scale, c.path, c.tiles, a, f.out.data_ptr(), lse, stream);
  return f;
}

// The status of a forward inside autograd travels in `Call` (a failed call is then repeated by the
// Python front, which raises).
struct SharedCall : torch::CustomClassHolder {
  Call c;
  int status = 0;
};

struct NaFunction : torch::autograd::Function<NaFunction> {
  // in: q, k, v and, where there are any, the extra keys and values
  static variable_list forward(AutogradContext* ctx, at::TensorList in,
                               const c10::intrusive_ptr<SharedCall>& call) {
    at::AutoDispatchBelowADInplaceOrView below;
    const bool extra = in.size() == 5;
    Forward f = forward_now(call->c, in[0], in[1], in[2], extra ? in[3] : Tensor(),
                            extra ? in[4] : Tensor(), true);
    call->status = f.status;
    variable_list saved{f.out, f.lse};
    saved.insert(saved.end(), in.begin(), in.end());
    ctx->save_for_backward(saved);
    ctx->saved_data["call"] = c10::IValue::make_capsule(call);
    ctx->set_materialize_grads(false);   // no zeros for the logsumexp's (ignored) gradient
    return {f.out, f.lse};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const auto call = c10::static_intrusive_pointer_cast<SharedCall>(
        ctx->saved_data["call"].toCapsule());
    variable_list g;
    {
      at::AutoDispatchBelowADInplaceOrView below;
      // only the logsumexp was differentiated: zeros
      g = gradients(call->c, saved, grads[0].defined() ? grads[0] : at::zeros_like(saved[0]));
    }
    g.emplace_back();
    return seal(std::move(g));
  }
  static variable_list gradients(const Call& c, const variable_list& s, const Tensor& d_out_) {
    // (saved-tensor hooks may have put them into other strides)
    const Tensor out = s[0].contiguous(), lse = s[1].contiguous();
    const Tensor &q = s[2], &k = s[3], &v = s[4];
    const bool extra = s.size() == 7;
    const Tensor ak = extra ? s[5] : Tensor(), av = extra ? s[6] : Tensor();
    c10::cuda::CUDAGuard guard(q.device());
    Problem p = c.p;
    if (c.dense) {
      p.nd = 1;
      p.shape = {(int)token_count(q), 1, 1};
      p.kernel = {p.shape[0], 1, 1};
      p.stride = p.dilation = {1, 1, 1};
      p.causal = {c.p.causal[0], 0, 0};
    }
    Tiles t;
    const bool tc = backward_on_tensor_cores(p, c.z, extra, &t) && p.kernel[0] >= 2;
    View qv, kv, vv;
    if (tc && !exact_gradients(p, extra)) {
      qv = as_view(q); kv = as_view(k); vv = as_view(v);
    } else {   // also exact ones: rows may be done again on the CUDA cores, which read no views
      qv = {q.contiguous(), 0}; kv = {k.contiguous(), 0}; vv = {v.contiguous(), 0};
    }
    const Tensor d_out = tc ? aligned(d_out_) : d_out_.contiguous();
    const Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(k.sizes(), q.options()),
                 dv = at::empty(k.sizes(), q.options());
    Tensor akc, avc, dak, dav;
    if (extra) {
      akc = ak.contiguous();
      avc = av.contiguous();
      dak = at::empty(ak.sizes(), q.options());
      dav = at::empty(ak.sizes(), q.options());
    }
    const Tensor delta = at::empty(lse.sizes(), lse.options());
    auto ptr = [](const Tensor& x) -> void* { return x.defined() ? x.data_ptr() : nullptr; };
    const Pointers a{qv.t.data_ptr(), kv.t.data_ptr(), vv.t.data_ptr(), qv.ts, kv.ts, vv.ts, ptr(akc),
                     ptr(avc), extra ? (int)ak.size(1) : 0};
    const GradPointers gp{dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), 0, 0, 0, ptr(dak), ptr(dav)};
    run_backward(p, c.z, c.scale, tc, t, a, out.data_ptr(), d_out.data_ptr(), lse.data_ptr<float>(), gp,
                 delta.data_ptr<float>(), stream_of(q));
    if (extra) return {dq, dk, dv, dak, dav};
    return {dq, dk, dv};
  }
};

// ---- a whole layer: projection, attention on the slices of its output, projection ----------------

Pointers slices_of(const Tensor& qkv, int H, int D) {
  const long long row = 3ll * H * D;
  uint8_t* base = static_cast<uint8_t*>(qkv.data_ptr());
  const int64_t step = (int64_t)H * D * qkv.element_size();
  return {base, base + step, base + 2 * step, row, row, row, nullptr, nullptr, 0};
}
struct LayerForward {
  Tensor qkv, attn, lse, y;
  int status;
};
LayerForward layer_now(const Call& c, const Tensor& x, const Tensor& w1, const Tensor& b1,
                       const Tensor& w2, const Tensor& b2, bool want_lse) {
  LayerForward f;
  c10::cuda::CUDAGuard guard(x.device());
  c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
  const auto opt = [](const Tensor& t) { return t.defined() ? std::optional<Tensor>(t) : std::nullopt; };
  f.qkv = at::linear(x, w1, opt(b1)).contiguous();
  f.attn = at::empty(x.sizes(), x.options());
  if (want_lse) {
    std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
    s.back() = c.z.Hq;
    f.lse = at::empty(s, x.options().dtype(at::kFloat));
  }
  f.status = run_forward(c.p, c.z, c.scale, c.path, c.tiles, slices_of(f.qkv, c.z.Hq, c.z.D),
                         f.attn.data_ptr(), want_lse ? f.lse.data_ptr<float>() : nullptr, stream_of(x));
  // not run: the layer goes through its modules then, and what an autograd node returns is dropped
  f.y = f.status == B200NA_OK ? at::linear(f.attn, w2, opt(b2)) : at::empty_like(x);
  return f;
}
// Bias gradient: column sums of the output gradient.
Tensor column_sum(const Tensor& m, int dt) {
  const Tensor out = at::empty({m.size(1)}, m.options());
  const Tensor scratch = at::empty({lib.column_sum_scratch(m.size(0), (int)m.size(1))},
                                   m.options().dtype(at::kByte));
  check(lib.column_sum(m.data_ptr(), out.data_ptr(), m.size(0), (int)m.size(1), dt, scratch.data_ptr(),
                       stream_of(m)),
        "b200na_column_sum");
  launches += 2;
  return out;
}

struct LayerFunction : torch::autograd::Function<LayerFunction> {
  // in: x, the two weights and the biases there are (`b1_at`, `b2_at`: their places, 0 = none)
  static Tensor forward(AutogradContext* ctx, at::TensorList in, int64_t b1_at, int64_t b2_at,
                        const c10::intrusive_ptr<SharedCall>& call) {
    at::AutoDispatchBelowADInplaceOrView below;
    const Tensor &x = in[0], &w1 = in[1], &w2 = in[2];
    LayerForward f = layer_now(call->c, x, w1, b1_at ? in[b1_at] : Tensor(), w2,
                               b2_at ? in[b2_at] : Tensor(), true);
    ctx->saved_data["b1"] = b1_at;
    ctx->saved_data["b2"] = b2_at;
    call->status = f.status;
    ctx->save_for_backward({x, w1, w2, f.qkv, f.attn, f.lse});
    ctx->saved_data["call"] = c10::IValue::make_capsule(call);
    return f.y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto s = ctx->get_saved_variables();
    const auto call = c10::static_intrusive_pointer_cast<SharedCall>(
        ctx->saved_data["call"].toCapsule());
    const Call& c = call->c;
    const Tensor &x = s[0], &w1 = s[1], &w2 = s[2];
    // (saved-tensor hooks may have put them into other strides)
    const Tensor qkv = s[3].contiguous(), attn = s[4].contiguous(), lse = s[5].contiguous();
    const int64_t b1_at = ctx->saved_data["b1"].toInt(), b2_at = ctx->saved_data["b2"].toInt();
    const bool need_x = ctx->needs_input_grad(0), need_w1 = ctx->needs_input_grad(1),
               need_w2 = ctx->needs_input_grad(2), need_b1 = b1_at && ctx->needs_input_grad(b1_at),
               need_b2 = b2_at && ctx->needs_input_grad(b2_at);
    variable_list g(3 + (b1_at != 0) + (b2_at != 0) + 3);   // and the three plain arguments
    {
      at::AutoDispatchBelowADInplaceOrView below;
      c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
      c10::cuda::CUDAGuard guard(x.device());
      const int64_t E = x.size(-1), T = x.numel() / E;
      const Tensor dy = aligned(grads[0]).view({T, E});
      if (need_w2) g[2] = at::mm(dy.t(), attn.view({T, E}));
      if (need_b2) g[b2_at] = column_sum(dy, c.z.dt);
      if (need_x || need_w1 || need_b1) {
        const Tensor d_attn = at::mm(dy, w2);
        const Tensor dqkv = at::empty({T, 3 * E}, x.options());
        const Tensor delta = at::empty(lse.sizes(), lse.options());
        Tiles t;
        const bool tc = backward_on_tensor_cores(c.p, c.z, false, &t);
        TORCH_CHECK(tc, "natten_b200: layer backward without tensor-core tiles");
        const Pointers d = slices_of(dqkv, c.z.Hq, c.z.D);
        const GradPointers gp{const_cast<void*>(d.q), const_cast<void*>(d.k), const_cast<void*>(d.v),
                              d.q_ts, d.k_ts, d.v_ts, nullptr, nullptr};
        run_backward(c.p, c.z, c.scale, tc, t, slices_of(qkv, c.z.Hq, c.z.D), attn.data_ptr(),
                     d_attn.data_ptr(), lse.data_ptr<float>(), gp, delta.data_ptr<float>(), stream_of(x));
        if (need_x) g[0] = at::mm(dqkv, w1).view(x.sizes());
        if (need_w1) g[1] = at::mm(dqkv.t(), x.contiguous().view({T, E}));
        if (need_b1) g[b1_at] = column_sum(dqkv, c.z.dt);
      }
    }
    return seal(std::move(g));
  }
};

// ---- arguments ------------------------------------------------------------------------------------

// An eager call on plain dense CUDA tensors: no tensor subclass, no function transform, no mode.
bool plain_mode() {
  const auto& tls = c10::impl::tls_local_dispatch_key_set();
  constexpr c10::DispatchKeySet kModes({c10::DispatchKey::Python, c10::DispatchKey::PythonDispatcher,
                                        c10::DispatchKey::PythonTLSSnapshot,
                                        c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                        c10::DispatchKey::FuncTorchDynamicLayerBackMode,
                                        c10::DispatchKey::FuncTorchVmapMode,
                                        c10::DispatchKey::Functionalize});
  return !tls.included_.has_any(kModes) && at::impl::PythonTorchFunctionTLS::stack_len() == 0 &&
         !torch::jit::tracer::isTracing();
}
bool plain_tensor(PyObject* o, Tensor* out) {
  if (!THPVariable_CheckExact(o)) return false;
  const Tensor& t = THPVariable_Unpack(o);
  constexpr c10::DispatchKeySet kOdd({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                                      c10::DispatchKey::FuncTorchBatched,
                                      c10::DispatchKey::FuncTorchGradWrapper,
                                      c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                      c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor});
  if (!t.is_cuda() || t.layout() != at::kStrided || t.is_nested() || t.key_set().has_any(kOdd))
    return false;
  if (t.unsafeGetTensorImpl()->has_symbolic_sizes_strides() || t._fw_grad(0).defined()) return false;
  *out = t;
  return true;
}
bool parse_int(PyObject* o, int minimum, int* out) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  const long v = PyLong_AsLongAndOverflow(o, &overflow);
  if (overflow || v < minimum || v > 0x7fffffff) return false;
  *out = (int)v;
  return true;
}
// an int for all axes or a tuple / list of nd ints; None = `fallback` (0: not allowed)
bool parse_dims(PyObject* o, int nd, int minimum, int fallback, std::array<int, kMaxDim>* out) {
  if (o == Py_None && fallback > 0) {
    for (int a = 0; a < nd; ++a) (*out)[a] = fallback;
    return true;
  }
  if (PyTuple_Check(o) || PyList_Check(o)) {
    if (PySequence_Fast_GET_SIZE(o) != nd) return false;
    for (int a = 0; a < nd; ++a)
      if (!parse_int(PySequence_Fast_GET_ITEM(o, a), minimum, &(*out)[a])) return false;
    return true;
  }
  int v;
  if (!parse_int(o, minimum, &v)) return false;
  for (int a = 0; a < nd; ++a) (*out)[a] = v;
  return true;
}
bool parse_flags(PyObject* o, int nd, std::array<int, kMaxDim>* out) {
  if (o == Py_None || PyBool_Check(o)) {
    for (int a = 0; a < nd; ++a) (*out)[a] = o == Py_True;
    return true;
  }
  if (!(PyTuple_Check(o) || PyList_Check(o)) || PySequence_Fast_GET_SIZE(o) != nd) return false;
  for (int a = 0; a < nd; ++a) {
    PyObject* x = PySequence_Fast_GET_ITEM(o, a);
    if (!PyBool_Check(x)) return false;
    (*out)[a] = x == Py_True;
  }
  return true;
}
// None or 0: D^-0.5
bool parse_scale(PyObject* o, int D, float* out) {
  double s = 0.;
  if (o != Py_None) {
    if (!PyFloat_CheckExact(o) && !PyLong_CheckExact(o)) return false;
    s = PyFloat_AsDouble(o);
    if (s == -1. && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
  }
  if (s == 0.) s = std::pow((double)D, -0.5);
  *out = (float)s;
  return *out > 0.f;
}
// The rules of the tensor checks in checks.py; `axes` token axes must match between q and k / v.
bool fits(const Tensor& q, const Tensor& k, const Tensor& v, int nd, bool same_tokens, Sizes* z) {
  if (q.dim() != nd + 3 || k.dim() != nd + 3 || v.dim() != nd + 3) return false;
  if (q.scalar_type() != k.scalar_type() || q.scalar_type() != v.scalar_type()) return false;
  if (q.device() != k.device() || q.device() != v.device()) return false;
  if (k.sizes() != v.sizes() || q.size(0) != k.size(0) || q.size(-1) != k.size(-1)) return false;
  for (int a = 0; a < nd; ++a) {
    if (q.size(1 + a) < 1 || k.size(1 + a) < 1 || q.size(1 + a) > 0x7fffffff ||
        k.size(1 + a) > 0x7fffffff)
      return false;
    if (same_tokens && q.size(1 + a) != k.size(1 + a)) return false;
  }
  const int64_t hq = q.size(-2), hk = k.size(-2), D = q.size(-1), B = q.size(0);
  if (B < 1 || hk < 1 || hq < hk || hq % hk || D < 1 || D > 256 || B > 0x7fffffff || hq > 0x7fffffff)
    return false;
  *z = {(int)B, (int)hq, (int)hk, (int)D, dtype_code(q.scalar_type())};
  return z->dt >= 0;
}
bool parse_problem(PyObject* kernel, PyObject* stride, PyObject* dilation, PyObject* causal, int nd,
                   c10::IntArrayRef shape, Problem* p) {
  p->nd = nd;
  if (!parse_dims(kernel, nd, 2, 0, &p->kernel) || !parse_dims(stride, nd, 1, 1, &p->stride) ||
      !parse_dims(dilation, nd, 1, 1, &p->dilation) || !parse_flags(causal, nd, &p->causal))
    return false;
  for (int a = 0; a < nd; ++a) {
    p->shape[a] = (int)shape[1 + a];
    if ((long long)p->kernel[a] * p->dilation[a] > p->shape[a] || p->stride[a] > p->kernel[a])
      return false;
  }
  return true;
}
PyObject* wrap(const Tensor& out, const Tensor& lse, bool want_lse) {
  if (!want_lse) return THPVariable_Wrap(out);
  PyObject* o = THPVariable_Wrap(out);
  PyObject* l = THPVariable_Wrap(lse);
  PyObject* t = PyTuple_New(2);
  PyTuple_SET_ITEM(t, 0, o);
  PyTuple_SET_ITEM(t, 1, l);
  return t;
}

bool any_requires_grad(std::initializer_list<const Tensor*> ts) {
  if (!c10::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}
// Runs a call that has passed every check, with autograd when a gradient is wanted.
PyObject* finish(const Call& c, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ak,
                 const Tensor& av, bool want_lse) {
  Tensor out, lse;
  if (any_requires_grad({&q, &k, &v, &ak, &av})) {
    if (is_8bit(c.z.dt)) Py_RETURN_NONE;   // no gradients for 8-bit operands
    auto call = c10::make_intrusive<SharedCall>();
    call->c = c;
    variable_list r;
    {
      pybind11::gil_scoped_release no_gil;
      const std::array<Tensor, 5> in{q, k, v, ak, av};
      r = NaFunction::apply(at::TensorList(in.data(), ak.defined() ? 5 : 3), call);
    }
    if (call->status != B200NA_OK) Py_RETURN_NONE;
    out = r[0];
    lse = r[1];
  } else {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    Forward f = forward_now(c, q, k, v, ak, av, want_lse);
    out = f.status == B200NA_OK ? f.out : Tensor();
    lse = f.lse;
  }
  if (!out.defined()) Py_RETURN_NONE;
  return wrap(out, lse, want_lse);
}
bool dense_taken(const Sizes& z) {
  if (reads_natively(z.dt, z.D)) return true;
  if (is_8bit(z.dt) || (is_16bit(z.dt) && z.D < 128)) return false;   // refused / padded first
  return true;
}

// na(nd, query, key, value, kernel_size, stride, dilation, is_causal, scale, additional_keys,
//    additional_values, return_lse)
PyObject* py_na(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 12, "na() takes 12 arguments");
  const int nd = (int)PyLong_AsLong(a[0]);
  Tensor q, k, v, ak, av;
  Call c;
  if (!plain_mode() || !plain_tensor(a[1], &q) || !plain_tensor(a[2], &k) || !plain_tensor(a[3], &v) ||
      !fits(q, k, v, nd, true, &c.z) ||
      !parse_problem(a[4], a[5], a[6], a[7], nd, q.sizes(), &c.p) ||
      !parse_scale(a[8], c.z.D, &c.scale))
    Py_RETURN_NONE;
  const bool extra = a[9] != Py_None || a[10] != Py_None;
  if (extra) {
    if (!plain_tensor(a[9], &ak) || !plain_tensor(a[10], &av) || ak.dim() != 4 || av.dim() != 4 ||
        ak.sizes() != av.sizes() || ak.size(0) != c.z.B || ak.size(1) < 1 || ak.size(1) > 0x7fffffff ||
        ak.size(2) != c.z.Hkv || ak.size(3) != c.z.D || ak.scalar_type() != q.scalar_type() ||
        av.scalar_type() != q.scalar_type() || ak.device() != q.device() || av.device() != q.device())
      Py_RETURN_NONE;
  }
  bool whole = !extra;
  for (int i = 0; i < nd; ++i)
    whole = whole && c.p.kernel[i] == c.p.shape[i] && (nd == 1 || !c.p.causal[i]);
  if (whole) {   // a window over the whole layout is dense attention
    long long tokens = 1;
    for (int i = 0; i < nd; ++i) tokens *= c.p.shape[i];
    if (!dense_taken(c.z) || tokens > 0x7fffffff) Py_RETURN_NONE;
    c.dense = true;
  } else {
    c.path = forward_path(c.p, c.z, ak.defined(), &c.tiles);
    if (c.path == Path::kNone) Py_RETURN_NONE;
  }
  return finish(c, q, k, v, ak, av, a[11] == Py_True);
  END_HANDLE_TH_ERRORS
}

// attention(query, key, value, is_causal, scale, return_lse)
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 6, "attention() takes 6 arguments");
  Tensor q, k, v;
  Call c;
  if (!plain_mode() || !plain_tensor(a[0], &q) || !plain_tensor(a[1], &k) || !plain_tensor(a[2], &v) ||
      !fits(q, k, v, 1, false, &c.z) || !PyBool_Check(a[3]) || !parse_scale(a[4], c.z.D, &c.scale) ||
      !dense_taken(c.z))
    Py_RETURN_NONE;
  c.p.causal[0] = a[3] == Py_True;
  c.dense = true;
  if (q.size(1) != k.size(1) && (c.p.causal[0] || any_requires_grad({&q, &k, &v}))) Py_RETURN_NONE;
  return finish(c, q, k, v, Tensor(), Tensor(), a[5] == Py_True);
  END_HANDLE_TH_ERRORS
}

// layer(nd, x, qkv_weight, qkv_bias, proj_weight, proj_bias, heads, kernel_size, stride, dilation,
//       is_causal, scale)
PyObject* py_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 12, "layer() takes 12 arguments");
  const int nd = (int)PyLong_AsLong(a[0]);
  Tensor x, w1, b1, w2, b2;
  Call c;
  if (!plain_mode() || at::autocast::is_autocast_enabled(at::kCUDA) || !plain_tensor(a[1], &x) ||
      !plain_tensor(a[2], &w1) || (a[3] != Py_None && !plain_tensor(a[3], &b1)) ||
      !plain_tensor(a[4], &w2) || (a[5] != Py_None && !plain_tensor(a[5], &b2)))
    Py_RETURN_NONE;
  const int heads = (int)PyLong_AsLong(a[6]);
  if (x.dim() != nd + 2 || heads < 1 || x.size(-1) % heads) Py_RETURN_NONE;
  const int64_t E = x.size(-1);
  const int dt = dtype_code(x.scalar_type());
  for (const Tensor* t : {&w1, &b1, &w2, &b2})
    if (t->defined() && (t->scalar_type() != x.scalar_type() || t->device() != x.device()))
      Py_RETURN_NONE;
  if (!is_16bit(dt) || E > 0x3fffffff || w1.dim() != 2 || w1.size(0) != 3 * E || w1.size(1) != E ||
      w2.dim() != 2 || w2.size(0) != E || w2.size(1) != E ||
      (b1.defined() && (b1.dim() != 1 || b1.size(0) != 3 * E)) ||
      (b2.defined() && (b2.dim() != 1 || b2.size(0) != E)))
    Py_RETURN_NONE;
  for (int i = 0; i <= nd; ++i)
    if (x.size(i) < 1 || x.size(i) > 0x7fffffff) Py_RETURN_NONE;
  c.z = {(int)x.size(0), heads, heads, (int)(E / heads), dt};
  if (!reads_natively(dt, c.z.D) ||
      !parse_problem(a[7], a[8], a[9], a[10], nd, x.sizes(), &c.p) ||
      !parse_scale(a[11], c.z.D, &c.scale))
    Py_RETURN_NONE;
  bool whole = true;
  for (int i = 0; i < nd; ++i)
    whole = whole && c.p.kernel[i] == c.p.shape[i] && (nd == 1 || !c.p.causal[i]);
  if (whole) Py_RETURN_NONE;
  c.path = forward_path(c.p, c.z, false, &c.tiles);
  if (c.path != Path::kTensorCore) Py_RETURN_NONE;
  Tensor y;
  if (any_requires_grad({&x, &w1, &b1, &w2, &b2})) {
    Tiles t;
    // exact gradients need contiguous operands: the layer in parts copies them
    if (!backward_on_tensor_cores(c.p, c.z, false, &t) || exact_gradients(c.p, false)) Py_RETURN_NONE;
    auto call = c10::make_intrusive<SharedCall>();
    call->c = c;
    {
      pybind11::gil_scoped_release no_gil;
      variable_list in{x, w1, w2};
      if (b1.defined()) in.push_back(b1);
      if (b2.defined()) in.push_back(b2);
      y = LayerFunction::apply(at::TensorList(in), b1.defined() ? 3 : 0, b2.defined() ? (int64_t)in.size() - 1 : 0, call);
    }
    if (call->status != B200NA_OK) Py_RETURN_NONE;
  } else {
    pybind11::gil_scoped_release no_gil;
    at::AutoDispatchBelowADInplaceOrView below;
    LayerForward f = layer_now(c, x, w1, b1, w2, b2, false);
    if (f.status == B200NA_OK) y = f.y;
  }
  if (!y.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(y);
  END_HANDLE_TH_ERRORS
}

// tiles(backward, shape, kernel, stride, dilation, is_causal[, extra]) -> (q tile, kv tile); with
// `extra` (whether there are extra tokens) the plan of the entries for views
PyObject* py_tiles(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK((n == 6 || n == 7) && PyTuple_Check(a[1]) && PyTuple_GET_SIZE(a[1]) >= 1 && PyTuple_GET_SIZE(a[1]) <= 3,
              "tiles(backward, shape, kernel, stride, dilation, is_causal)");
  Problem p;
  p.nd = (int)PyTuple_GET_SIZE(a[1]);
  TORCH_CHECK(parse_dims(a[1], p.nd, 1, 0, &p.shape) && parse_dims(a[2], p.nd, 1, 0, &p.kernel) &&
                  parse_dims(a[3], p.nd, 1, 0, &p.stride) && parse_dims(a[4], p.nd, 1, 0, &p.dilation) &&
                  parse_flags(a[5], p.nd, &p.causal),
              "tiles(): expected tuples of positive integers and flags");
  const bool backward = a[0] == Py_True;
  const Tiles t = n == 7 ? plan(p, backward, a[6] == Py_True)
                         : (backward ? choose_backward(p) : choose_forward(p));
  PyObject* out = PyTuple_New(2);
  for (int i = 0; i < 2; ++i) {
    PyObject* x = PyTuple_New(p.nd);
    for (int d = 0; d < p.nd; ++d) PyTuple_SET_ITEM(x, d, PyLong_FromLong(i ? t.kv[d] : t.q[d]));
    PyTuple_SET_ITEM(out, i, x);
  }
  return out;
  END_HANDLE_TH_ERRORS
}

PyObject* py_init(PyObject*, PyObject* path) {
  HANDLE_TH_ERRORS
  const char* p = PyUnicode_AsUTF8(path);
  TORCH_CHECK(p, "init(path)");
  void* h = dlopen(p, RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h, "cannot load ", p, ": ", dlerror());
#define X(name)                                                                    \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, "b200na_" #name));      \
  TORCH_CHECK(lib.name, p, " has no b200na_" #name);
  B200NA_FUNCTIONS(X)
#undef X
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}
PyObject* py_launches(PyObject*, PyObject*) { return PyLong_FromLongLong(launches.load()); }

PyMethodDef methods[] = {
    {"init", py_init, METH_O, "Binds the C library at `path`."},
    {"launches", py_launches, METH_NOARGS, "Kernel launches issued through this module so far."},
    {"na", (PyCFunction)(void*)py_na, METH_FASTCALL, nullptr},
    {"attention", (PyCFunction)(void*)py_attention, METH_FASTCALL, nullptr},
    {"layer", (PyCFunction)(void*)py_layer, METH_FASTCALL, nullptr},
    {"tiles", (PyCFunction)(void*)py_tiles, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "torch_binding", nullptr, -1, methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_torch_binding() { return PyModule_Create(&module_def); }
