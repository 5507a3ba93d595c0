// noalloc.cu -- y = A x on caller-owned device buffers, allocating nothing.
//
// Some callers cannot let a library allocate device memory: a host
// application that hands all of HBM to its own pool allocator at start-up
// (a further cudaMalloc fails or breaks its accounting), or code that must
// not take the device-wide synchronisation that cudaMalloc / cudaFree imply
// in the middle of a latency-critical loop.
// pdlp_spmv_noalloc serves them: the caller passes the CSR matrix and the
// vectors already in device memory, and the only scratch the product needs
// (per-tile partial sums of rows that cross tile boundaries, and an error
// flag) lives in the file-scope device array below, which every GPU that
// loads this library holds until the process exits.
//
// Tiles are cut at fixed non-zero offsets, so no row plan has to be built or
// stored.  A thread of a block loads the columns and values of kRun consecutive
// non-zeros (16 bytes a load where the caller's arrays are aligned), gathers x
// and keeps the products' factors in registers; two of the block's warps look up
// the rows that start in the tile meanwhile (32 row pointers a step).  The rows
// then mark where they start, and each thread folds its non-zeros run by run --
// a run is one row's share of them -- with one FMA a product, so that none is
// rounded by itself; the runs meet in shared memory, where a thread adds those
// of each row, or a warp where there are more than kShort.  A row that continues
// past its tile leaves one partial per tile in the scratch array, and a second
// kernel adds them in a fixed order, so the result is bitwise reproducible.
//
// Bound by the gathers of x and by each tile's round trips.  Through the entry
// point, against a thread adding each row from both factors in shared memory:
// 20M non-zeros with power-law columns 358 -> 145 us, a transport matrix (rows
// of 2,000 and 5,000) 1,280 -> 141 us (2.3 TB/s of matrix and vectors), 10M in
// rows of 34 185 -> 94 us, of 65 184 -> 95 us; 20k non-zeros 35 -> 33 us, which
// is launches and the read of the error flag.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <mutex>
#include <string>

#include "common.cuh"
#include "pdlp_gb300.h"

namespace {

constexpr int kTile = 2048;  // non-zeros per thread block
constexpr int kRun = kTile / pdlp::kThreads;  // consecutive non-zeros of a thread
static_assert(kRun == 8, "a thread's row marks are one 8-byte word");
constexpr int kMaxTiles = PDLP_NOALLOC_MAX_TILES;

// Scratch of every call: own[t] (partial of the row that starts in tile t and
// runs past it), in[t] (partial of the row that reached tile t from an
// earlier tile), own_row[t] (that row, or -1), and the error flag.
struct Scratch {
  double own[kMaxTiles];
  double in[kMaxTiles];
  int own_row[kMaxTiles];
  int error[2];  // of this call, and of the next one (cleared by this one)
};

static __device__ __align__(256) Scratch g_scratch;

// Runs of a row that one thread adds (up to 512 products); beyond, its adds in
// turn take longer than a warp's, whose tree of shuffles costs 5 FP64 issue slots
// of 16 cycles.  10M non-zeros in rows of 65: 94 us with 64 or 16, 181 with 8.
constexpr int kShort = 64;

// First r in [0, rows) with ptr[r] >= key, else rows, by a warp: each step
// keeps the one of 33 parts that the answer is in.
__device__ __forceinline__ int lower_bound_rows(const int *ptr, int rows, int key) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = rows;  // the answer is in [lo, hi]
  while (hi > lo) {
    const long n = hi - lo;
    const int at = lo + (int)(n * (lane + 1) / 33);
    const unsigned below = __ballot_sync(0xffffffffu, at < hi && ptr[at] < key);
    // a malformed (unsorted) ptr still ends: the interval shrinks every step
    const int k = below ? 32 - __clz(below) : 0;  // probes 0 .. k - 1 taken as below
    const int next_lo = k ? lo + (int)(n * k / 33) + 1 : lo;
    const int next_hi = k < 32 ? min(hi, lo + (int)(n * (k + 1) / 33)) : hi;
    lo = min(next_lo, hi);
    hi = max(next_hi, lo);
  }
  return lo;
}

// Sum of the runs of [lo, hi) by a warp, in a fixed order: sp[lo] and sp at the
// multiples of kRun above it, below hi.  Every lane returns it.
__device__ __forceinline__ double warp_runs(const double *sp, int lo, int hi) {
  const int first = lo / kRun;  // run of lo
  double s = 0.0;
#pragma unroll 4
  for (int g = first + (int)(threadIdx.x & 31); g * kRun < hi; g += 32)
    s += sp[g == first ? lo : g * kRun];
  return pdlp::warp_sum(s);
}

// 5 blocks per SM: 6 spill (powerlaw 155 us), 4 leave too few loads in flight
// (156 us).  Row marks are bytes: as bits, set by atomics, rows of one entry took
// 107 us instead of 94 (5M of them).
__global__ void __launch_bounds__(pdlp::kThreads, 5)
    k_spmv_tiles(int rows, int cols, int nnz, int ntiles, const int *__restrict__ ptr,
                 const int *__restrict__ col, const double *__restrict__ val,
                 const double *__restrict__ x, double *__restrict__ y, Scratch *s, int slot) {
  __shared__ double sp[kTile];  // sums of runs, each where its run starts
  __shared__ __align__(8) unsigned char starts[kTile];  // 1: a row starts here
  __shared__ int s_rows[2];
  const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k0 = t * kTile;
  const int k1 = min(nnz, k0 + kTile);
  const int len = k1 > k0 ? k1 - k0 : 0;
  const int mine = tid * kRun, n = min(kRun, len - mine);  // this thread's elements
  int c[kRun];
  double v[kRun];
  const bool aligned =
      ((reinterpret_cast<uintptr_t>(col) | reinterpret_cast<uintptr_t>(val)) & 15) == 0;
  if (aligned && n == kRun) {
#pragma unroll
    for (int u = 0; u < kRun; u += 4) {
      const int4 q = __ldcs(reinterpret_cast<const int4 *>(col + k0 + mine + u));
      c[u] = q.x; c[u + 1] = q.y; c[u + 2] = q.z; c[u + 3] = q.w;
    }
#pragma unroll
    for (int u = 0; u < kRun; u += 2) {
      const double2 q = __ldcs(reinterpret_cast<const double2 *>(val + k0 + mine + u));
      v[u] = q.x; v[u + 1] = q.y;
    }
  } else {
#pragma unroll
    for (int u = 0; u < kRun; ++u) {
      c[u] = 0;
      v[u] = 0.0;
      if (u < n) {
        c[u] = __ldcs(col + k0 + mine + u);
        v[u] = __ldcs(val + k0 + mine + u);
      }
    }
  }
  if (warp < 2) {
    const bool first = warp == 0;
    int r = first ? 0 : rows;
    if (first ? t > 0 : t < ntiles - 1) r = lower_bound_rows(ptr, rows, first ? k0 : k1);
    if (lane == 0) s_rows[warp] = r;
  }
  reinterpret_cast<unsigned long long *>(starts)[tid] = 0ull;
  if (tid == 0) {
    if (t == 0 && (ptr[0] != 0 || ptr[rows] != nnz)) atomicOr(&s->error[slot], 1);
    if (t == 0) s->error[slot ^ 1] = 0;
    s->own_row[t] = -1;  // set below by the row that runs past k1, if any
  }
  // row pointers are validated over all rows (grid-stride), so a malformed
  // CSR always raises the flag; every access below stays in bounds either way
  for (long r = (long)t * pdlp::kThreads + tid; r < rows; r += (long)ntiles * pdlp::kThreads)
    if (ptr[r] > ptr[r + 1]) atomicOr(&s->error[slot], 1);
  bool bad = false;
  double g[kRun];
#pragma unroll
  for (int u = 0; u < kRun; ++u) {
    const bool in = c[u] >= 0 && c[u] < cols;
    if (u < n) bad |= !in;  // flagged, never dereferenced
    g[u] = u < n && in ? __ldg(x + c[u]) : 0.0;
  }
  if (bad) atomicOr(&s->error[slot], 2);
  __syncthreads();
  const int rA = s_rows[0], rB = s_rows[1];
#pragma unroll 1
  for (int r = rA + tid; r < rB; r += pdlp::kThreads) {
    const int a = ptr[r] - k0;
    if (a >= 0 && a < len) starts[a] = 1;
  }
  __syncthreads();
  {
    // the runs among this thread's elements, each left where it starts; bit u of
    // `here`: a row starts at element u (the lowest bits of the eight bytes)
    const unsigned long long bytes = reinterpret_cast<const unsigned long long *>(starts)[tid];
    const unsigned here = (unsigned)((bytes * 0x0102040810204080ull) >> 56);
    double sum = 0.0;
    int from = mine;
#pragma unroll
    for (int u = 0; u < kRun; ++u) {
      if (u > 0 && ((here >> u) & 1u)) {
        sp[from] = sum;
        sum = 0.0;
        from = mine + u;
      }
      if (u < n) sum = fma(v[u], g[u], sum);
    }
    sp[from] = sum;
  }
  __syncthreads();
  // rows starting in this tile; the one running past k1 leaves its partial
  for (int base = rA + 32 * warp; base < rB; base += pdlp::kThreads) {
    const int r = base + lane;
    int a = 0, e = 0;
    bool live = r < rB;
    if (live) {
      a = ptr[r];
      e = ptr[r + 1];
      live = a <= e && a >= k0 && e <= nnz;  // else flagged by the validation loop
    }
    const int lo = a - k0, hi = live ? min(e, k1) - k0 : lo;
    double sum = 0.0;
    const int runs = hi > lo ? (hi - 1) / kRun - lo / kRun + 1 : 0;
    if (runs > 0 && runs <= kShort) {
      sum = sp[lo];
#pragma unroll 4
      for (int q = (lo / kRun + 1) * kRun; q < hi; q += kRun) sum += sp[q];
    }
    unsigned todo = __ballot_sync(0xffffffffu, runs > kShort);
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1;
      const double w = warp_runs(sp, __shfl_sync(0xffffffffu, lo, src),
                                 __shfl_sync(0xffffffffu, hi, src));
      if (lane == src) sum = w;
    }
    if (live) {
      if (e > k1) {
        s->own[t] = sum;
        s->own_row[t] = r;
      } else {
        y[r] = sum;
      }
    }
  }
  // partial of the row (started in an earlier tile) that runs into this one
  if (warp == pdlp::kThreads / 32 - 1) {
    double in = 0.0;
    if (t > 0 && rA > 0) in = warp_runs(sp, 0, min(ptr[rA], k1) - k0);  // it ends where rA starts
    if (lane == 0) s->in[t] = in;
  }
}

// y[r] for a row crossing tiles: its own partial plus the partials of the
// tiles it runs into, in tile order (a warp's lanes take turns over more than
// 32 of them)
__global__ void k_spmv_tiles_fix(int ntiles, const int *__restrict__ ptr, double *__restrict__ y,
                                 const Scratch *__restrict__ s) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  int r = -1, count = 0;
  if (t < ntiles) r = s->own_row[t];
  if (r >= 0) {
    const long end = ((long)ptr[r + 1] + kTile - 1) / kTile;  // first tile past the row
    count = (int)max(0l, min((long)ntiles, end) - (t + 1));
  }
  double tot = r >= 0 ? s->own[t] : 0.0;
  if (count <= 32)
    for (int u = 1; u <= count; ++u) tot += s->in[t + u];
  unsigned todo = __ballot_sync(0xffffffffu, count > 32);
  while (todo) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    const int n = __shfl_sync(0xffffffffu, count, src), from = __shfl_sync(0xffffffffu, t, src);
    double w = 0.0;
    for (int u = 1 + lane; u <= n; u += 32) w += s->in[from + u];
    w = pdlp::warp_sum(w);
    if (lane == src) tot += w;
  }
  if (r >= 0) y[r] = tot;
}

// Device address of the scratch array, per device.  Only a successful
// lookup is kept: a lookup that failed (say, before the device could be
// used) is tried again by the next call.
constexpr int kMaxDevices = 64;
Scratch *g_addr[kMaxDevices] = {};
unsigned g_calls[kMaxDevices] = {};  // the error slot alternates
std::mutex g_addr_mu;

thread_local std::string g_err;

int fail(int code, const std::string &msg) {
  g_err = msg;
  fprintf(stderr, "[cupdlpx-gb300] pdlp_spmv_noalloc: %s\n", msg.c_str());
  return code;
}

}  // namespace

extern "C" const char *pdlp_spmv_noalloc_error(void) { return g_err.c_str(); }

extern "C" int pdlp_spmv_noalloc(int rows, int cols, int nnz, const int *row_ptr,
                                 const int *col_ind, const double *vals, const double *x,
                                 double *y, void *stream) {
  if (rows < 0 || cols < 0 || nnz < 0)
    return fail(-1, "negative size");
  const long ntiles_l = nnz > 0 ? ((long)nnz + kTile - 1) / kTile : 1;
  if (ntiles_l > kMaxTiles)
    return fail(-3, "nnz " + std::to_string(nnz) + " exceeds the maximum of " +
                        std::to_string((long)kMaxTiles * kTile) +
                        " non-zeros (PDLP_NOALLOC_MAX_TILES tiles of 2048)");
  if (rows == 0) {
    if (nnz > 0) return fail(-1, "non-zeros given for a matrix without rows");
    return 0;
  }
  if (!row_ptr || !y || (nnz > 0 && (!col_ind || !vals || !x)))
    return fail(-1, "NULL buffer");
  const int ntiles = (int)ntiles_l;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= kMaxDevices)
    return fail(-2, std::string("no usable CUDA device: ") + cudaGetErrorString(e));
  // set-up, once per device, with that device current
  Scratch *s = nullptr;
  int slot = 0;
  {
    std::lock_guard<std::mutex> lk(g_addr_mu);
    if (!g_addr[dev]) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, g_scratch);
      if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return fail(-2, std::string("cudaGetSymbolAddress failed: ") + cudaGetErrorString(e));
      }
      g_addr[dev] = (Scratch *)p;
    }
    s = g_addr[dev];
    slot = (int)(g_calls[dev] & 1u);
  }
  cudaStream_t st = (cudaStream_t)stream;
  // this call's error flag was cleared by the call before it (at first by the
  // array's initialisation); every other slot a call reads, the same call
  // writes first
  k_spmv_tiles<<<ntiles, pdlp::kThreads, 0, st>>>(rows, cols, nnz, ntiles, row_ptr, col_ind,
                                                  vals, x, y, s, slot);
  if (ntiles > 1)  // no row leaves a single tile
    k_spmv_tiles_fix<<<(ntiles + pdlp::kThreads - 1) / pdlp::kThreads, pdlp::kThreads, 0, st>>>(
        ntiles, row_ptr, y, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    cudaMemsetAsync(s->error, 0, sizeof(s->error), st);  // the kernel that clears it did not run
    return fail(-2, std::string("launch: ") + cudaGetErrorString(e));
  }
  int flag = 0;
  e = cudaMemcpyAsync(&flag, &s->error[slot], sizeof(int), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(-2, std::string("sync: ") + cudaGetErrorString(e));
  {
    std::lock_guard<std::mutex> lk(g_addr_mu);
    ++g_calls[dev];  // the kernel has run, so the other slot is clear
  }
  if (flag & 2) return fail(-4, "column index out of range");
  if (flag & 1) return fail(-4, "malformed row pointers");
  return 0;
}
