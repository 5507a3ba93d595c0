// strip.cuh -- the sparse matrix format of the solver and its product kernel.
//
// Replaces the reference's cusparseSpMV(CSR_ALG2) calls
// (src/pdlp_core_op.cu:501-504, :534-537, :671-674, :801-804;
// src/utils.cu:134-140, :645-653, :750-758) and the element kernels after
// them, as spmv.cuh does on plain CSR.
//
// The upload orders the rows of A and of A^T (the constraints and the
// variables) by decreasing length, stably, and the solve works in that order
// throughout; only its inputs and results are permuted (the layout is SELL-C-sigma,
// Kreutzer et al. 2014, with slices of 32 and all rows sorted).  Then
//   * rows of at most kStripRow non-zeros form strips of 32 consecutive rows
//     of (nearly) one length, stored element-major: element k of the strip's
//     rows is 32 consecutive columns and values.  A warp takes a strip, a
//     lane a row: every load of the matrix and of the per-row vectors is
//     coalesced, a row's sum stays in its lane's registers (no shared memory,
//     no barrier, no cross-lane sum), and the epilogue runs with all lanes.
//     GB300 issues one FP64 warp instruction per 16 cycles and SM whatever
//     lanes are active, so the one FMA per non-zero and the full epilogues
//     are what an FP64 product can cost least.  A matrix with too few rows
//     to give the chip's warps a strip each has 2, 4 or 8 lanes to a row (and
//     16, 8 or 4 rows to a strip): there the time is the chain of a strip's
//     loads (about 1,300 cycles for four elements), not the issue slots;
//   * rows of up to kWideRow have 8 lanes each in strips of their own (wide
//     strips, which stand before the others), or 16 or 32 in a small matrix:
//     one reduction over 8 lanes for four rows instead of one over 32 for each;
//   * longer rows come first (the front), in CSR order: a warp takes items of
//     consecutive rows of together up to kStripItem non-zeros (lanes stride a
//     row, its lane sums are added across lanes in FP64, and the item's rows
//     run their epilogues together), one row of up to twice as many in a large
//     front, or an eighth of a chunk of a longer row
//     (32 of every 256 elements), whose sums are added in order by the last
//     one to finish (atomic ticket).
// Shorter rows of a strip are padded with column -1, which is skipped.
// Items and strips are dealt to the warps of a fixed grid in a fixed order,
// so every sum has a fixed order and results are bitwise reproducible.
//
// FP32 sums.  An FP32 solve's path depends on the rounding of its sums (the
// 20M-non-zero power-law LP takes 55,200 or 69,400 iterations to 1e-4 with two
// orders of the same products), so FP32 matrices keep the order that the fused
// kernel gives them, or the FP32 pairs of the pipelined one (strip_pairs below:
// by the lengths of all rows, so that one long row changes nothing for the
// others): a row's elements are folded in segments that end at
// fixed distances from the start of the row's tile of that kernel's plan, and
// the segments are added in order.  StripPlan::sums holds, per row, the
// segment length and the row's phase in it, or the number of lanes that the
// kernel strides a long row with.
#pragma once

#include <limits.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "spmv.cuh"
#include "spmv_pipe.cuh"

namespace pdlp {

constexpr int kStripRow = 64;     // longest row of a strip
constexpr int kWideRow = 256;     // longest row of a wide strip
constexpr int kStripItem = 1024;  // non-zeros of a front item (of several rows)
constexpr int kNarrow = 2;        // elements of a narrow matrix's strips

struct StripPlan {
  int on = 0;                  // the matrix is stored in this format
  int nfront = 0;              // rows longer than kWideRow (they come first)
  int nwide = 0, wide_end = 0; // wide strips and the end of their rows
  int nitem = 0, nlong = 0, nstrip = 0;
  int lg = 0, lgw = 0;         // a strip's (wide strip's) rows have 1 << lg lanes each
  // reduction partials: one per strip, whatever warp took it, for LPs that a
  // team may run (team.cuh); else one per block
  int unit_parts = 0;
  int pairs = 0;               // FP32 sums in pairs (see above)
  int narrow = 0;              // strips of up to kNarrow elements only, a lane a row
  int grid = 0;                // blocks of the product kernel (8 items or strips each)
  long store = 0;              // stored elements, padding included
  int *off = nullptr;          // strip s: 32-element columns off[s] .. off[s + 1]
  // {first row, rows, first element, end}, or for 32 of every 256 elements of
  // a chunk of a long row {row, -(long id + 1), first element, chunk end}
  int4 *item = nullptr;
  int2 *lrow = nullptr;        // per long row {first item, items}
  const unsigned char *sums = nullptr;  // per row, for FP32 matrices (StripHost::sums)
  unsigned *lcnt = nullptr;    // per long row arrival counter (per solve, kept at 0)
  double *lsum = nullptr;      // per item: its sum (per solve)
};

struct StripHost {
  std::vector<int> perm;       // position -> original row (empty: the same)
  std::vector<int> fptr;       // element offsets of the front's rows
  std::vector<int4> item;
  std::vector<int2> lrow;
  std::vector<int> off;
  int nwide = 0, wide_end = 0;
  int lg = 0, lgw = 0;
  long store = 0;
};

// Strip s of a matrix: the lanes of its rows, its first row and the end of the
// rows of its kind.
struct StripPlace {
  int lg, row, end;
};
__host__ __device__ inline StripPlace strip_place(const StripPlan &p, int rows, int s) {
  if (s < p.nwide) return {p.lgw, p.nfront + s * (32 >> p.lgw), p.wide_end};
  return {p.lg, p.wide_end + (s - p.nwide) * (32 >> p.lg), rows};
}

// Lanes of a row (as their logarithm): as many as keep the strips within 8
// warps of each of `sms` SMs.
inline int strip_lanes(long rows, int sms, int least = 0, int most = 3) {
  int lg = least;
  while (lg < most && (rows << (lg + 1)) <= 32L * 8 * sms) ++lg;
  return lg;
}

// FP32 sum of a row: low 4 bits the phase, high 4 the segment length; or
// kSumStrided + log2(lanes).
constexpr int kSumStrided = 0xF0;

// Per row of a CSR matrix, from the tiles of the fused kernel (tile and chunk
// as its plan) ...
inline void strip_sums_fused(int rows, const int *ptr, int tile, int chunk,
                             std::vector<unsigned char> &sums) {
  std::vector<int4> blk;
  std::vector<int2> lrow;
  build_plan_host(rows, ptr, tile, blk, lrow, chunk);
  const bool direct = tile == 1024 && rows > 0 && plan_direct(blk, ptr[rows]);
  sums.assign(rows, 0);
  for (const int4 &b : blk) {
    const int R = b.y - b.x, len = b.w - b.z;
    if (b.y < 0) {
      sums[b.x] = kSumStrided + 8;
    } else if (R > 1 && len <= 64 * R) {
      const int seg = direct && len >= kDirectMinAvg * R ? 4 : 8;
      const int from = seg == 4 ? b.z & ~3 : b.z;
      for (int r = b.x; r < b.y; ++r)
        sums[r] = (unsigned char)((ptr[r] - from) % seg | seg << 4);
    } else {
      int g = 8;  // one row: all 256 threads
      if (R > 1)
        for (g = 0; (2 << g) <= kThreads / R && g < 5;) ++g;
      for (int r = b.x; r < b.y; ++r) sums[r] = (unsigned char)(kSumStrided + g);
    }
  }
}

// Whether an FP32 matrix is summed in pairs: one of kPairsMinNnz non-zeros or
// more, unless more than a twentieth of them lie in rows that the pipelined
// kernel takes at a loss -- alone in a tile they do not fill (more than
// kPipeMedRows, up to kPipeFill entries) or in chunks.  Those two kernels' times
// draw the line; above it a matrix keeps the pairs it has had there, below it
// the fused kernel's sums.  Pipelined over fused, FP32 dual step: random rows of
// 10 to 100 0.71-0.95, of 120 (a quarter of the non-zeros in rows above 128)
// 1.9-2.0, of 160 1.8; uniform rows of 130 2.0, 300 1.06, 350 0.86, 500 0.88,
// 800 0.65, 2,000 0.92, 2,100 2.0, 5,000 1.6; columns of power-law LPs 1.6-2.2.
constexpr long kPairsMinNnz = 1L << 22;
constexpr int kPipeFill = 340;
inline bool strip_pairs(int rows, const int *ptr) {
  const long nnz = rows > 0 ? ptr[rows] : 0;
  if (nnz < kPairsMinNnz) return false;
  long loss = 0;
  for (int r = 0; r < rows; ++r) {
    const int len = ptr[r + 1] - ptr[r];
    if ((len > kPipeMedRows && len <= kPipeFill) || len > kPipeTile) loss += len;
  }
  return 20 * loss <= nnz;
}

// ... or of the pipelined kernel (nv row vectors staged; its one-row tiles are
// summed in pairs too, where the order hardly matters).
inline void strip_sums_pipe(int rows, const int *ptr, int nv, std::vector<unsigned char> &sums) {
  std::vector<int4> blk;
  std::vector<int2> lrow;
  build_pipe_plan_host(rows, ptr, nv, blk, lrow);
  sums.assign(rows, 15 << 4);
  for (const int4 &b : blk) {
    if (b.y - b.x < 2) continue;
    const int seg = ((b.w - b.z + kThreads - 1) / kThreads) | 1;
    for (int r = b.x; r < b.y; ++r) sums[r] = (unsigned char)((ptr[r] - b.z) % seg | seg << 4);
  }
}

// Host: order and cut the rows of a CSR matrix; tile: the longest row that the
// fused kernel does not cut, chunk: elements of a long row's chunk (a multiple
// of 256).
inline void build_strip_host(int rows, const int *ptr, int sms, int tile, int chunk,
                             StripHost &h) {
  h = StripHost();
  h.lg = strip_lanes(rows, sms);
  // stable order by decreasing length: the front by sorting, the rest by
  // counting
  std::vector<int> front;
  std::vector<int> count(kWideRow + 2, 0);
  bool sorted = true;
  for (int r = 0, before = INT_MAX; r < rows; ++r) {
    const int len = ptr[r + 1] - ptr[r];
    sorted &= len <= before;
    before = len;
    if (len > kWideRow) front.push_back(r);
    else ++count[kWideRow - len + 1];
  }
  const int nfront = (int)front.size();
  h.wide_end = nfront;
  for (int l = 1; l <= kWideRow - kStripRow; ++l) h.wide_end += count[l];
  h.lgw = strip_lanes(h.wide_end - nfront, sms, 3, 5);
  if (!sorted) {
    h.perm.resize(rows);
    std::stable_sort(front.begin(), front.end(), [&](int a, int b) {
      return ptr[a + 1] - ptr[a] > ptr[b + 1] - ptr[b];
    });
    std::copy(front.begin(), front.end(), h.perm.begin());
    count[0] = nfront;
    for (int l = 1; l <= kWideRow + 1; ++l) count[l] += count[l - 1];
    for (int r = 0; r < rows; ++r) {
      const int len = ptr[r + 1] - ptr[r];
      if (len <= kWideRow) h.perm[count[kWideRow - len]++] = r;
    }
  }
  // front: items and chunks.  Items of a small front are smaller, down to a
  // row each: as many as keep them within 8 warps of each SM (a transport LP
  // of 854 x 94, 800 FP64 iterations and the set-up: 22.0 -> 17.4 ms)
  h.fptr.assign(1, 0);
  for (int i = 0; i < nfront; ++i)
    h.fptr.push_back(h.fptr.back() + ptr[front[i] + 1] - ptr[front[i]]);
  const int most = std::min(kStripItem, h.fptr.back() / (8 * sms));
  // a row of more than this is cut: in a large front, whose rows fill the chip as
  // they are, only above twice an item (5,300 rows of 1,500, FP32 dual step 0.061
  // -> 0.043 ms: no sums to store and count); in a small one all rows that the
  // fused kernel cuts too, so that a warp's rounds of loads are few
  const int whole = std::max(tile, std::min(2 * kStripItem, h.fptr.back() / (8 * sms)));
  for (int i = 0; i < nfront;) {
    const int a = h.fptr[i], e = h.fptr[i + 1];
    if (e - a > whole) {
      h.lrow.push_back(make_int2((int)h.item.size(), 0));
      for (int k = a; k < e; k += chunk) {
        const int end = std::min(k + chunk, e);
        for (int j = k; j < std::min(k + 256, end); j += 32) {
          h.item.push_back(make_int4(i, -(int)h.lrow.size(), j, end));
          ++h.lrow.back().y;
        }
      }
      ++i;
    } else {
      const int i0 = i;
      do ++i;
      while (i < nfront && i - i0 < 32 && h.fptr[i + 1] - a <= most);
      h.item.push_back(make_int4(i0, i - i0, a, h.fptr[i]));
    }
  }
  // strips
  long at = ((long)h.fptr.back() + 31) / 32;
  auto strips = [&](int begin, int end, int lanes) {
    for (int r = begin; r < end; r += 32 / lanes) {
      h.off.push_back((int)at);
      const int first = sorted ? r : h.perm[r];  // its longest row
      at += (ptr[first + 1] - ptr[first] + lanes - 1) / lanes;
    }
  };
  strips(nfront, h.wide_end, 1 << h.lgw);
  h.nwide = (int)h.off.size();
  strips(h.wide_end, rows, 1 << h.lg);
  h.off.push_back((int)at);
  h.store = at * 32;
}

// One matrix as the kernels read it (arrays of `store` elements; ptr: the
// front's rows).
template <class M>
struct StripMat {
  const int *ptr, *col;
  const M *val;
  int rows;
  StripPlan p;
};

// Matrix data: read once a sweep from HBM (evict first), or kept in L2 by LPs
// that fit there.
template <bool STREAM, class T>
__device__ __forceinline__ T ld_matrix(const T *p) {
  if constexpr (STREAM) return __ldcs(p);
  else return __ldg(p);
}

// A strip row's running sum in its lane.  FP64: two independent chains, so that
// a lane waits for half of its row's additions; one for rows of two, where the
// chains' addition would take as long and an issue slot more.
template <class M, bool PAIR>
struct StripSum {
  double s[2] = {0.0, 0.0};
  __device__ __forceinline__ explicit StripSum(int) {}
  __device__ __forceinline__ void add(bool second, double a, double x) {
    if (second) s[1] = fma(a, x, s[1]);
    else s[0] = fma(a, x, s[0]);
  }
  __device__ __forceinline__ double total(bool both) const { return both ? s[0] + s[1] : s[0]; }
};
// FP32: segment by segment (see above); PAIR: each in an FP32 pair.
template <bool PAIR>
struct StripSum<float, PAIR> {
  using Acc = typename std::conditional<PAIR, LaneAcc<float>, float>::type;
  Acc seg{}, all{};
  int left, len;  // elements until the segment ends, its length
  __device__ __forceinline__ explicit StripSum(int how) {
    len = how >> 4;
    if (len == 15 && !PAIR) len = 8;
    left = len - (how & 15);
    if (left <= 0) left = len;
    if constexpr (!PAIR) all = -0.f;  // -0 + s is s
  }
  __device__ __forceinline__ void end() {
    if constexpr (PAIR) {
      all.add_pair(seg.hi(), seg.lo());
      seg = LaneAcc<float>();
    } else {
      all += seg;
      seg = 0.f;
    }
  }
  __device__ __forceinline__ void add(bool, float a, float x) {
    if (left == 0) {
      end();
      left = len;
    }
    --left;
    if constexpr (PAIR) seg.add(a, x);
    else seg = fmaf(a, x, seg);
  }
  __device__ __forceinline__ float total(bool) {
    end();
    if constexpr (PAIR) return isfinite(all.lo()) ? all.rounded() : all.hi();
    else return all;
  }
  // pairs of a row's lanes, after total()
  __device__ __forceinline__ float across(int lanes) {
    for (int o = 1; o < lanes; o <<= 1) {
      const float h = __shfl_xor_sync(0xffffffffu, all.hi(), o);
      const float l = __shfl_xor_sync(0xffffffffu, all.lo(), o);
      all.add_pair(h, l);
    }
    return isfinite(all.lo()) ? all.rounded() : all.hi();
  }
};

template <class Epi, class M>
__device__ __forceinline__ void strip_epilogue(const Epi &epi, int row, M sum,
                                               const typename pre_of<Epi>::type &pre,
                                               double *acc) {
  if constexpr (has_preload<Epi>::value) epi.row_pre(row, sum, pre, acc);
  else epi.row(row, sum, acc);
}

// Four elements of a strip's lanes.
template <class M>
struct StripQuad {
  int c[4];
  M v[4];
};
template <bool STREAM, class M>
__device__ __forceinline__ void strip_load(const int *col, const M *val, int left,
                                           StripQuad<M> &q) {
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    q.c[u] = -1;
    q.v[u] = M(0);
    if (u < left) {
      q.c[u] = ld_matrix<STREAM>(col + u * 32);
      q.v[u] = ld_matrix<STREAM>(val + u * 32);
    }
  }
}

// The start of a strip (a team loads its next one before it waits).
template <class M>
struct StripHead {
  int o0, n;
  StripQuad<M> q;
};
template <bool STREAM, int MOST = 4, class M>
__device__ __forceinline__ void strip_head(const StripMat<M> &A, int s, StripHead<M> &x) {
  x.o0 = x.n = 0;
  if (s < A.p.nstrip) {
    x.o0 = __ldg(A.p.off + s);
    x.n = __ldg(A.p.off + s + 1) - x.o0;
  }
  const size_t at = (size_t)x.o0 * 32 + (threadIdx.x & 31);
  strip_load<STREAM>(A.col + at, A.val + at, MOST < 4 ? min(x.n, MOST) : x.n, x.q);
}

// Sums of the strip rows (FP32) that the fused kernel strides with several
// lanes (see "FP32 sums"), by the whole warp, row by row: its lanes take those
// lanes' parts of the row.  total: this lane's row's sum.  Such a row stands
// beside long ones or alone at the end of that kernel's tile: 637 of the 2M
// columns of the power-law LP, 513 of them with one entry (any order).
template <bool STREAM, class Epi>
__device__ __forceinline__ void strip_strided(const Epi &epi, const int *col, const float *val,
                                              int n, int lg, bool mine, int how, float &total) {
  const int lane = threadIdx.x & 31;
  unsigned todo = __ballot_sync(0xffffffffu, mine && how >= kSumStrided);
#pragma unroll 1
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int lanes = 1 << (__shfl_sync(0xffffffffu, how, src) - kSumStrided);
    double t = 0.0;
#pragma unroll 1
    for (int j = lane; j < lanes && j < n << lg; j += 32) {
      float s = 0.f;
#pragma unroll 1
      for (int e = j; e < n << lg; e += lanes) {
        // element e of the row whose first lane is src (col, val: lane 0's)
        const int at = (e >> lg) * 32 + src + (e & ((1 << lg) - 1));
        const int c = ld_matrix<STREAM>(col + at);
        if (c >= 0) s = fmaf(ld_matrix<STREAM>(val + at), epi.gather(c), s);
      }
      t += (double)s;
    }
    t = warp_sum(t);
    if (lane == src) total = (float)t;
  }
}

// Sum of this lane's row in a wide strip (FP32) where the fused kernel strides it
// with at least its 1 << lg lanes here: element k of lane j is element (k << lg) + j
// of the row, so that a lane's elements are those of one, two or four of the fused
// kernel's lanes in turn, or, of 256, of a lane each.
template <bool STREAM, class Epi>
__device__ __forceinline__ float strip_wide_strided(const Epi &epi, const int *col,
                                                    const float *val, int n, int lg, int how) {
  const int turns = 1 << max(0, how - kSumStrided - lg);  // the fused kernel's lanes of a lane
  float s[4] = {};
  double t = 0.0;
#pragma unroll 1
  for (int k = 0; k < n; k += 4) {
    StripQuad<float> q;
    strip_load<STREAM>(col + k * 32, val + k * 32, n - k, q);
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q.c[u] >= 0) x[u] = epi.gather(q.c[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q.c[u] >= 0) {
        if (turns > 4) t += (double)fmaf(q.v[u], x[u], 0.f);
        else if (turns == 4) s[u] = fmaf(q.v[u], x[u], s[u]);
        else if (turns == 2) s[u & 1] = fmaf(q.v[u], x[u], s[u & 1]);
        else s[0] = fmaf(q.v[u], x[u], s[0]);
      }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) t += (double)s[u];
  for (int o = 1; o < (1 << lg); o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return (float)t;
}

// Sum of this lane's row in a wide strip (FP32, not in pairs), by the row's 1 << lg
// lanes: a lane folds every (1 << lg)th segment, eight elements' loads at a time,
// and the segments are added in order.  Element by element, every lane of the row
// would add all of them with three shuffles each.  col, val: of the row's first
// lane.
template <bool STREAM, class Epi>
__device__ __forceinline__ float strip_segments(const Epi &epi, const int *col, const float *val,
                                                int n, int lg, int how) {
  const int lane = threadIdx.x & 31, G = 1 << lg, base = lane & ~(G - 1);
  const int len = how >= kSumStrided ? 8 : how >> 4, phase = how >= kSumStrided ? 0 : how & 15;
  const int all_elements = n << lg;
  // rounds of the row with the most segments in the strip
  const int rounds = (all_elements + 7 + 3) / 4 / G + 1;
  float all = -0.f;
#pragma unroll 1
  for (int r = 0; r < rounds; ++r) {
    const int first = (r * G + lane - base) * len - phase;
    float s = 0.f;
    bool any = false;
    constexpr int U = 4;
#pragma unroll
    for (int h = 0; h < 8; h += U) {
      int c[U];
      float v[U], x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int e = first + h + u;
        c[u] = -1;
        if (h + u < len && e >= 0 && e < all_elements) {
          const int at = (e >> lg) * 32 + (e & (G - 1));
          c[u] = ld_matrix<STREAM>(col + at);
          v[u] = ld_matrix<STREAM>(val + at);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c[u] >= 0) x[u] = epi.gather(c[u]);
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (c[u] >= 0) {
          s = fmaf(v[u], x[u], s);
          any = true;
        }
    }
    const unsigned real = __ballot_sync(0xffffffffu, any);
    if (real == 0u) break;
    for (int g = 0; g < G; ++g) {
      const float add = __shfl_sync(0xffffffffu, s, base + g);
      if ((real >> (base + g)) & 1u) all += add;
    }
  }
  return all;
}

// Strip s, by a warp; `head` as strip_head loaded it.  NARROW: of a narrow matrix;
// WIDE: of a matrix that may have wide strips.
template <bool STREAM, bool PAIR, bool NARROW = false, bool WIDE = !NARROW, class Epi, class M>
__device__ __forceinline__ void strip_rows(const StripMat<M> &A, const Epi &epi, double *acc,
                                           int s, const StripHead<M> &head) {
  const int lane = threadIdx.x & 31, o0 = head.o0, n = head.n;
  StripQuad<M> q = head.q;
  // the row of this lane, and whether it is the lane that ends the row
  const StripPlace place =
      WIDE ? strip_place(A.p, A.rows, s)
           : StripPlace{A.p.lg, A.p.nfront + s * (32 >> A.p.lg), A.rows};
  const int lg = NARROW ? 0 : place.lg, row = place.row + (lane >> lg);
  const bool ends = row < place.end && (lane & ((1 << lg) - 1)) == 0;
  const int *col = A.col + (size_t)o0 * 32 + lane;
  const M *val = A.val + (size_t)o0 * 32 + lane;
  typename pre_of<Epi>::type pre;
  if constexpr (has_preload<Epi>::value)
    if (ends) epi.preload(row, pre);
  int how = 0;
  if constexpr (sizeof(M) == 4) how = row < A.rows ? __ldg(A.p.sums + row) : 8 << 4;
  if constexpr (sizeof(M) == 4 && !PAIR && WIDE)
    if (s < A.p.nwide) {
      const int up = lane & ((1 << lg) - 1);
      const bool strided = how >= kSumStrided;
      M total = M(0);
      if (__any_sync(0xffffffffu, !strided))
        total = strip_segments<STREAM>(epi, col - up, val - up, n, lg, how);
      if (__any_sync(0xffffffffu, strided)) {
        const M t = strip_wide_strided<STREAM>(epi, col, val, n, lg, how);
        if (strided) total = t;
        strip_strided<STREAM>(epi, col - lane, val - lane, n, lg,
                              ends && how - kSumStrided < lg, how, total);
      }
      if (ends) strip_epilogue(epi, row, total, pre, acc);
      return;
    }
  StripSum<M, PAIR> sum(how);
  // four elements ahead, but not in FP32 kernels that stream: at their 40
  // registers it spills (power-law dual step 0.088 ms ahead, 0.053 without;
  // FP64 0.083 ahead, 0.087 without)
  constexpr bool kAhead = (sizeof(M) == 8 || !STREAM) && !NARROW;
  constexpr int kLoad = NARROW ? kNarrow : 4;
#pragma unroll 1
  for (int k = 0; k < (NARROW ? 1 : n); k += 4) {
    M x[kLoad];
    // padding: no load, and 0 times the padding's 0
#pragma unroll
    for (int u = 0; u < kLoad; ++u) {
      x[u] = M(0);
      if (q.c[u] >= 0) x[u] = epi.gather(q.c[u]);
    }
    StripQuad<M> next;
    if constexpr (kAhead)
      strip_load<STREAM>(col + (k + 4) * 32, val + (k + 4) * 32, n - k - 4, next);
#pragma unroll
    for (int u = 0; u < kLoad; ++u) {
      if (k + u >= n) break;  // the same for every lane
      if (sizeof(M) == 8 || PAIR || lg == 0) {
        if (sizeof(M) == 8 || q.c[u] >= 0) sum.add(u % 2 && n > 2, q.v[u], x[u]);
      } else {
        // a row's elements in their order, by every lane of the row
        const int base = lane & ~((1 << lg) - 1);
        for (int g = 0; g < (1 << lg); ++g) {
          const M v = __shfl_sync(0xffffffffu, q.v[u], base + g);
          const M y = __shfl_sync(0xffffffffu, x[u], base + g);
          if (__shfl_sync(0xffffffffu, q.c[u], base + g) >= 0) sum.add(false, v, y);
        }
      }
    }
    if constexpr (kAhead)
      q = next;
    else if constexpr (!NARROW)
      strip_load<STREAM>(col + (k + 4) * 32, val + (k + 4) * 32, n - k - 4, q);
  }
  M total = sum.total(n > 2);
  if constexpr (sizeof(M) == 8)
    for (int o = 1; o < (1 << lg); o <<= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  if constexpr (sizeof(M) == 4 && PAIR)
    if (lg > 0) total = sum.across(1 << lg);
  if constexpr (sizeof(M) == 4 && !PAIR)
    if (n > 1 || lg > 0) strip_strided<STREAM>(epi, col - lane, val - lane, n, lg, ends, how, total);
  if (ends) strip_epilogue(epi, row, total, pre, acc);
}

// Sum, by a warp, of elements a + lane, a + lane + step, ... below e of a front
// row (every lane returns it): lane chains, across lanes in FP64.  The chains
// of an FP32 matrix are single ones in FP32, or pairs.
template <bool STREAM, bool PAIR, class Epi, class M>
__device__ __forceinline__ double strip_warp_sum(const StripMat<M> &A, const Epi &epi, int a,
                                                 int e, int step) {
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  LaneAcc<M> pair[2];
  M one = M(0);
#pragma unroll 1
  for (int k = a + lane; k < e; k += step * U) {
    int c[U];
    M v[U], x[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + step * u < e) {
        c[u] = ld_matrix<STREAM>(A.col + k + step * u);
        v[u] = ld_matrix<STREAM>(A.val + k + step * u);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + step * u < e) x[u] = epi.gather(c[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + step * u < e) {
        if constexpr (sizeof(M) == 4 && !PAIR) one = fmaf(v[u], x[u], one);
        else pair[u % 2].add(v[u], x[u]);
      }
  }
  if constexpr (sizeof(M) == 4 && !PAIR) {
    return warp_sum((double)one);
  } else {
    pair[0].add_pair(pair[1].hi(), pair[1].lo());
    return warp_sum(pair[0].total());
  }
}

// s plus the products of elements k, k + step, ... below e, in order.  Four
// elements' loads at a time: one by one each gather waits for its own column.
template <bool STREAM, class Epi>
__device__ __forceinline__ float strip_chain(const StripMat<float> &A, const Epi &epi, int k,
                                             int e, int step, float s) {
  constexpr int U = 4;
#pragma unroll 1
  for (; k < e; k += U * step) {
    int c[U];
    float v[U], x[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u * step < e) {
        c[u] = ld_matrix<STREAM>(A.col + k + u * step);
        v[u] = ld_matrix<STREAM>(A.val + k + u * step);
      }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u * step < e) x[u] = epi.gather(c[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (k + u * step < e) s = fmaf(v[u], x[u], s);
  }
  return s;
}

// Sum of the whole front row [a, e) as `how` says (FP32, see above).
template <bool STREAM, class Epi>
__device__ __forceinline__ float strip_row_sum(const StripMat<float> &A, const Epi &epi, int a,
                                               int e, int how) {
  const int lane = threadIdx.x & 31;
  if (how >= kSumStrided) {
    const int lanes = 1 << (how - kSumStrided);
    double t = 0.0;
    if (lanes <= 32) {
      if (lane < lanes) t = (double)strip_chain<STREAM>(A, epi, a + lane, e, lanes, 0.f);
    } else {
      // four of the lanes' chains side by side: a row that 256 lanes take has a
      // few elements for each
      constexpr int U = 4;
#pragma unroll 1
      for (int j = lane; j < lanes; j += 32 * U) {
        float s[U] = {};
#pragma unroll 1
        for (int k = a + j; k < e; k += lanes) {
          int c[U];
          float v[U], x[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j + 32 * u < lanes && k + 32 * u < e) {
              c[u] = ld_matrix<STREAM>(A.col + k + 32 * u);
              v[u] = ld_matrix<STREAM>(A.val + k + 32 * u);
            }
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j + 32 * u < lanes && k + 32 * u < e) x[u] = epi.gather(c[u]);
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (j + 32 * u < lanes && k + 32 * u < e) s[u] = fmaf(v[u], x[u], s[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) t += (double)s[u];
      }
    }
    return (float)warp_sum(t);
  }
  // segments: a lane each, added in order
  const int len = how >> 4, phase = how & 15;
  const int count = (e - a + phase + len - 1) / len;
  float all = -0.f;
  for (int j = 0; j < count; j += 32) {
    const int k0 = max(a, a - phase + (j + lane) * len), k1 = min(e, a - phase + (j + lane + 1) * len);
    const float s = strip_chain<STREAM>(A, epi, k0, k1, 1, 0.f);
    const int n = min(32, count - j);
    for (int g = 0; g < n; ++g) all += __shfl_sync(0xffffffffu, s, g);
  }
  return all;
}

// Front item i, by a warp; `chunk(i, b, sum)` takes the sum of a chunk of a
// long row (called by every lane).
template <bool STREAM, bool PAIR, class Epi, class M, class Chunk>
__device__ __forceinline__ void strip_front(const StripMat<M> &A, const Epi &epi, double *acc,
                                            int i, Chunk &&chunk) {
  const int lane = threadIdx.x & 31;
  const int4 b = __ldg(A.p.item + i);
  if (b.y < 0) {
    chunk(i, b, strip_warp_sum<STREAM, PAIR>(A, epi, b.z, b.w, 256));
    return;
  }
  typename pre_of<Epi>::type pre;
  int a = 0, e = 0;
  if (lane < b.y) {
    a = __ldg(A.ptr + b.x + lane);
    e = __ldg(A.ptr + b.x + lane + 1);
    if constexpr (has_preload<Epi>::value) epi.preload(b.x + lane, pre);
  }
  M mine = M(0);
#pragma unroll 1
  for (int r = 0; r < b.y; ++r) {
    const int ra = __shfl_sync(0xffffffffu, a, r), re = __shfl_sync(0xffffffffu, e, r);
    M t;
    if constexpr (sizeof(M) == 4 && !PAIR)
      t = strip_row_sum<STREAM>(A, epi, ra, re, __ldg(A.p.sums + b.x + r));
    else
      t = (M)strip_warp_sum<STREAM, PAIR>(A, epi, ra, re, 32);
    if (lane == r) mine = t;
  }
  if (lane < b.y) strip_epilogue(epi, b.x + lane, mine, pre, acc);
}

// Partials of one unit's reductions, by its warp.
template <int NF, unsigned MAXMASK, int NA>
__device__ __forceinline__ void strip_partials(double (&acc)[NA], double *part, int unit,
                                               int units) {
#pragma unroll
  for (int f = 0; f < NF; ++f)
    acc[f] = ((MAXMASK >> f) & 1u) ? warp_max(acc[f]) : warp_sum(acc[f]);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int f = 0; f < NF; ++f) part[(long)f * units + unit] = acc[f];
  }
}

// Partials of a block's: through shared memory, a warp for each reduction.  A
// shuffle tree in every warp costs 5 FP64 issue slots of 16 cycles per warp and
// reduction, more than the strips' own arithmetic in the three sums of a
// transport LP's evaluation; this takes 12 per block and reduction.
template <int NF, unsigned MAXMASK, int NA>
__device__ __forceinline__ void strip_block_partials(const double (&acc)[NA], double *part) {
  __shared__ double all[NF][kThreads];
  const int lane = threadIdx.x & 31, f = threadIdx.x >> 5;
#pragma unroll
  for (int g = 0; g < NF; ++g) all[g][threadIdx.x] = acc[g];
  __syncthreads();
  if (f >= NF) return;
  const bool most = (MAXMASK >> f) & 1u;
  double v = all[f][lane];
#pragma unroll
  for (int k = 32; k < kThreads; k += 32) {
    const double o = all[f][lane + k];
    v = most ? fmax(v, o) : v + o;
  }
  v = most ? warp_max(v) : warp_sum(v);
  if (lane == 0) part[(long)f * gridDim.x + blockIdx.x] = v;
}

// Epi as for spmv_fused (spmv.cuh).  A warp takes one item or strip, so that
// nothing but the kernel's parameters outlives a strip: in a loop over strips
// the compiler keeps a dozen vector pointers in registers (spills at 48), at
// the price of the gathers in flight.
// Bound by FP64 issue (16 cycles per warp instruction and SM) and by the
// gathers' L2 requests.  20M non-zeros, ms per launch inside a solve, before (the
// faster of the CSR kernels), with a block's warps far apart in the list, and
// now: power-law primal step 0.155, 0.147, 0.120 (FP32 0.106, 0.123, 0.107), dual
// step 0.128, 0.089, 0.084 (FP32 0.104, 0.057, 0.051); transport primal step
// 0.185, 0.206, 0.204 (FP32 0.132, 0.118, 0.118), dual step 0.108, 0.112, 0.096
// (FP32 0.084, 0.104, 0.074).  5 blocks per SM: 6 spill more (FP32 power-law
// primal step 0.139 against 0.132 ms; FP32 pairs, which need fewer registers, run
// at 6), 4 (no spills) took the transport primal step to 0.258.
// NARROW: the step kernels of a large matrix whose rows have at most two entries
// (a transport LP's columns).  There is no loop and nothing but one strip, so 8
// blocks fit an SM, and their vectors' loads are what such a step is: transport
// primal step 0.204 -> 0.201 ms (6 blocks 0.207), FP32 0.118 -> 0.096, FP32
// matrix 0.218 -> 0.181 (before the strips 0.185, 0.132 and 0.201).
// Blocks per SM the kernel's registers must allow.  Plain FP32 with wide strips
// spills 200 bytes at 5: 4 where the matrix stays in L2 (3M power-law non-zeros, FP32
// primal step 33 -> 24 us), 5 where it streams from HBM (20M: 107 us, 110 at 4).
template <bool FP64, bool STREAM, bool PAIR, bool NARROW, bool WIDE>
constexpr int strip_blocks() {
  return NARROW ? 8 : FP64 ? 5 : PAIR ? 6 : WIDE && !STREAM ? 4 : 5;
}

// WIDE: the matrix has wide strips; without them the plain FP32 kernels are spared
// their code, which takes registers from the other rows'.
template <class Epi, bool STREAM, bool PAIR, bool NARROW = false, bool WIDE = !NARROW>
__global__ void __launch_bounds__(
    kThreads, (strip_blocks<sizeof(typename Epi::val_t) == 8, STREAM, PAIR, NARROW, WIDE>()))
    spmv_strip(const __grid_constant__ StripMat<typename Epi::val_t> A,
               double *__restrict__ part, double *__restrict__ lpart, Epi epi) {
  using M = typename Epi::val_t;
  constexpr int NF = Epi::NF;
  __shared__ double sc[4];
  // a block's warps are neighbours in the list: of one length, so that none
  // holds the block's place on the SM for long, and with gathers in common
  const int w = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  const int units = A.p.nitem + A.p.nstrip;
  if (!epi.init()) return;
  if (threadIdx.x == 0) epi.prologue(sc);
  __syncthreads();
  epi.bind(sc);
  double acc[NF > 0 ? NF : 1];
#pragma unroll
  for (int f = 0; f < (NF > 0 ? NF : 1); ++f) acc[f] = 0.0;
  const int lane = threadIdx.x & 31;
  if constexpr (NARROW) {
    if (w < units) {
      StripHead<M> head;
      strip_head<STREAM, kNarrow>(A, w, head);
      strip_rows<STREAM, PAIR, true>(A, epi, acc, w, head);
    }
    if constexpr (NF > 0) strip_block_partials<NF, Epi::MAXMASK>(acc, part);
    return;
  }
  auto unit = [&](int i) {
    if (i >= A.p.nitem) {
      StripHead<M> head;
      strip_head<STREAM>(A, i - A.p.nitem, head);
      strip_rows<STREAM, PAIR, false, WIDE>(A, epi, acc, i - A.p.nitem, head);
      return;
    }
    strip_front<STREAM, PAIR>(A, epi, acc, i, [&](int at, const int4 &b, double sum) {
      if (lane != 0) return;
      const int lid = -b.y - 1;
      A.p.lsum[at] = sum;
      __threadfence();
      const int2 L = A.p.lrow[lid];
      if (atomicAdd(A.p.lcnt + lid, 1u) != (unsigned)L.y - 1u) return;
      __threadfence();
      double tot = 0.0;
#pragma unroll 4
      for (int c = 0; c < L.y; ++c) tot += __ldcg(A.p.lsum + L.x + c);
      double lacc[NF > 0 ? NF : 1];
#pragma unroll
      for (int f = 0; f < (NF > 0 ? NF : 1); ++f) lacc[f] = 0.0;
      epi.row(b.x, (M)tot, lacc);
      if constexpr (NF > 0) {
#pragma unroll
        for (int f = 0; f < NF; ++f) lpart[f * A.p.nlong + lid] = lacc[f];
      }
      A.p.lcnt[lid] = 0u;  // ready for the next launch
    });
  };
  if (w < units) unit(w);
  if constexpr (NF > 0) {
    if (A.p.unit_parts) {
      if (w < units) strip_partials<NF, Epi::MAXMASK>(acc, part, w, units);
      return;
    }
    strip_block_partials<NF, Epi::MAXMASK>(acc, part);
  }
}

}  // namespace pdlp
