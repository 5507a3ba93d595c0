// team.cuh -- whole PDHG iterations in one launch, by a team of CTAs.
//
// An LP of up to a few million non-zeros spends its time between kernels, not
// in them: with one launch per product an iteration of a 20,000-non-zero LP
// takes 11.8 us and a power iteration 22 us, of which the arithmetic is well
// under 1 us.  Here one cooperative launch runs hundreds of iterations: its
// CTAs (the team, one or two per SM) take the same strips of A and A^T
// throughout and meet at a barrier between a product and the next one that
// gathers its result.  Measured on GB300, that barrier costs 2,700 cycles
// (1.3 us) from 16 to 152 CTAs, so a team is spread over as many SMs as it
// has strips: GB300 issues one FP64 warp instruction per 16 cycles and SM.
//
// What is left is those barriers and, between them, the chain of a strip's
// loads.  Measured, whole solves: 20,000 non-zeros 34.6 -> 21.3 ms; a million
// 64 -> 35 ms (39 -> 21 us an iteration, 53 -> 28 us a power iteration).
//
// The strips are those of strip.cuh.  All orders are fixed by the plan, so
// results are bitwise reproducible and do not depend on what else runs.
#pragma once

#include <stdint.h>

#include <algorithm>

#include "bulk.cuh"
#include "strip.cuh"

namespace pdlp {

// LPs below this many non-zeros run their loop and power method as a resident
// team, where team_ctas finds one.
constexpr long kTeamMaxNnz = 1L << 22;
constexpr int kTeamThreads = kThreads;
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kTeamCtasPerSm = 2;

struct TeamBar {
  unsigned *count;  // arrivals so far (0 at launch)
  int *err;         // set when a wait ran out
};

struct TeamSmem {
  double red[8 * 8];
  unsigned target;  // arrivals the last barrier waited for (thread 0's)
  int ok;
};

// Barrier over the team: writes before it are visible after it.  False, in
// every thread of the CTA, when the wait ran out (kBulkWaitCycles, a constant: read
// from memory the limit costs a 40k x 100k LP 1.5 us an iteration): the caller
// returns, and the other CTAs' waits run out too.  The host then takes the
// launch's work back and repeats it with a kernel per product.
__device__ __forceinline__ bool team_sync(const TeamBar &b, TeamSmem &sm) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned target = sm.target + gridDim.x;
    sm.target = target;
    // release: orders the CTA's writes, which the block barrier put before it
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.count) : "memory");
    const long long t0 = clock64();
    int ok = 1;
    for (;;) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(b.count) : "memory");
      if ((int)(seen - target) >= 0) break;
      if (clock64() - t0 > kBulkWaitCycles) {
        atomicOr(b.err, 1);
        ok = 0;
        break;
      }
    }
    sm.ok = ok;
  }
  __syncthreads();
  return sm.ok != 0;
}

// The team's copy of its parameters, read where it is used: an index that the
// compiler cannot see through keeps it from hoisting a dozen pointers out of
// the loops that use them (they would fill the registers and spill).
template <class Data>
__device__ __forceinline__ const Data &team_data(const Data &data) {
  int zero = 0;
  asm volatile("" : "+r"(zero));
  return (&data)[zero];
}

// Strips are dealt to the CTAs in turn, so that an SM gets a second one only
// when every SM has one.
__device__ __forceinline__ int team_strip() {
  return (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
}
// One product with its epilogue, over the team.  `data` is the team's copy of
// its parameters in shared memory; mat(data) and make(data) give the matrix
// and the epilogue; `first` is the head of the warp's first strip,
// loaded before the barrier that the product waits for.  The epilogue's NF
// reductions leave the partials that the product's own kernel leaves
// (strip.cuh), so that a team and single launches compute the same bits.
// Nothing here takes the address of what lives across a barrier: local memory
// is read through the L1 that the barrier's acquire has just emptied.
template <int NF, unsigned MAXMASK, class Data, class Mat, class Make, class M>
__device__ __forceinline__ void team_phase(const Data &data, Mat mat, Make make, double *part,
                                           const StripHead<M> &first) {
  const int W = gridDim.x * kTeamWarps;
  int s = team_strip();
  StripHead<M> x = first;
  if (s >= mat(data).p.nstrip) return;
#pragma unroll 1
  for (;;) {
    const Data &here = team_data(data);
    double acc[NF > 0 ? NF : 1];
#pragma unroll
    for (int f = 0; f < (NF > 0 ? NF : 1); ++f) acc[f] = 0.0;
    strip_rows<false, false, false, Data::kWide>(mat(here), make(here), acc, s, x);
    if constexpr (NF > 0) strip_partials<NF, MAXMASK>(acc, part, s, mat(here).p.nstrip);
    s += W;
    if (s >= mat(here).p.nstrip) return;
    strip_head<false>(mat(here), s, x);
  }
}
template <int NF, unsigned MAXMASK, class Data, class Mat, class Make>
__device__ __forceinline__ void team_phase(const Data &data, Mat mat, Make make, double *part) {
  using M = std::remove_const_t<std::remove_pointer_t<decltype(mat(data).val)>>;
  StripHead<M> x;
  strip_head<false>(mat(data), team_strip(), x);
  team_phase<NF, MAXMASK>(data, mat, make, part, x);
}

// ------------------------------------------------------------- host side
// A solve in flight in this process (one of these per request).
struct SolveInFlight {
  SolveInFlight();
  ~SolveInFlight();
  SolveInFlight(const SolveInFlight &) = delete;
  SolveInFlight &operator=(const SolveInFlight &) = delete;
};
// The right to run a team.  A team is the fastest way through one small LP,
// but it occupies the SMs while it waits at its barriers: solves that run side
// by side get more done with a kernel per product (16 uneven LPs: 0.24 s
// against 0.46 s).  So a solve takes its turn only while it is the only one in
// flight, and looks again after every kTeamChunk iterations; both ways compute
// the same bits.  At most one team is in flight in the process: two could each
// hold part of the SMs and wait for the rest.
class TeamTurn {
 public:
  explicit TeamTurn(bool wanted);
  ~TeamTurn();
  TeamTurn(const TeamTurn &) = delete;
  TeamTurn &operator=(const TeamTurn &) = delete;
  explicit operator bool() const { return held_; }
  static bool alone();

 private:
  bool held_ = false;
};

// CTAs of the team for an LP's matrices; 0: no team.  A matrix with a front (rows
// of more than 256 entries) has none: its items have not been tried in a team as
// it is (an earlier one, with a barrier of their own for their sums, took 25 ms on
// a small LP of long rows, against 17 with a kernel per product).  Nor has one with more than
// two strips for a warp: the barriers no longer show beside the strips, but every
// CTA folds every strip's partial sums itself.  FP64, 600 iterations with set-up,
// team and single launches: 65k x 22k with 2 entries a row 15.1 and 17.2 ms, 131k
// x 44k 25.9 and 27.2, 262k x 87k 40.3 and 38.2, 524k x 175k 64 and 54, 4M x 1.3M
// 402 and 268; with 4M non-zeros throughout, 66k 75.4 and 73.8, 131k 134 and 131,
// 262k 150 and 138.
inline int team_ctas(long nnz, const StripPlan &A, const StripPlan &AT, int nsm) {
  if (nnz <= 0 || nnz >= kTeamMaxNnz || A.nitem > 0 || AT.nitem > 0) return 0;
  const int work = std::max(A.nstrip, AT.nstrip);
  if (work > 2 * nsm * kTeamCtasPerSm * kTeamWarps) return 0;
  // one CTA per SM until its warps have a strip each, then two
  return work <= nsm * kTeamWarps ? std::max(1, std::min(work, nsm)) : nsm * kTeamCtasPerSm;
}

// Sets a team's arrival counter for a launch: to 0, or, with PDLP_TEAM_FAIL=1, to
// a number from which no barrier completes, so that every wait runs out (as where
// the CTAs do not run at the same time for longer than that).
void team_reset(unsigned *count, cudaStream_t st);

// False when the device cannot hold the team's CTAs at once (an SM limit on
// the process, say): nothing was launched.
template <class... Params, class... Args>
bool team_launch(int ctas, void (*kernel)(Params...), cudaStream_t st, Args &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kTeamThreads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
    cudaGetLastError();
    return false;
  }
  PDLP_CUDA(e);
  return true;
}

}  // namespace pdlp
