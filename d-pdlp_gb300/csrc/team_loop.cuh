// team_loop.cuh -- the PDHG loop of one LP inside one launch (see team.cuh),
// included by solver_impl.cuh after the scalar logic it shares with the
// one-kernel-per-product path.
#pragma once

#include "team.cuh"

namespace pdlp {

// The step epilogues with the iteration's flags at run time.
template <class T, class M, bool FPE>
struct TeamPrimal {
  using val_t = M;
  using Pre = PrimalPre<T>;
  const Dev<T> &d;
  T tau, w, omw;
  int par;  // parity of the iteration: x[par] is the current iterate
  bool major;
  __device__ __forceinline__ M gather(int i) const { return (M)d.y[par][i]; }
  __device__ __forceinline__ void preload(int j, Pre &p) const {
    p.xc = d.x[par][j];
    p.c = d.c[j];
    p.lv = d.lv[j];
    p.uv = d.uv[j];
    p.x0 = d.x0[j];
  }
  __device__ __forceinline__ void row(int j, M s, double *acc) const {
    Pre p;
    preload(j, p);
    row_pre(j, s, p, acc);
  }
  __device__ __forceinline__ void row_pre(int j, M s, const Pre &p, double *acc) const {
    primal_update(d, j, (T)s, p, tau, w, omw, major, FPE, d.rho_is_one != 0,
                  d.x[par ^ 1], acc);
  }
};
template <class T, class M, bool FPE>
struct TeamDual {
  using val_t = M;
  using Pre = DualPre<T>;
  const Dev<T> &d;
  T sigma, inv_sigma, w, omw;
  int par;
  bool major;
  __device__ __forceinline__ M gather(int j) const { return (M)d.xref[j]; }
  __device__ __forceinline__ void preload(int i, Pre &p) const {
    p.yc = d.y[par][i];
    p.lc = d.lc[i];
    p.uc = d.uc[i];
    p.y0 = d.y0[i];
  }
  __device__ __forceinline__ void row(int i, M s, double *acc) const {
    Pre p;
    preload(i, p);
    row_pre(i, s, p, acc);
  }
  __device__ __forceinline__ void row_pre(int i, M s, const Pre &p, double *acc) const {
    dual_update(d, i, (T)s, p, sigma, inv_sigma, w, omw, major, FPE, d.rho_is_one != 0,
                d.y[par ^ 1], acc);
  }
};

struct TeamRun {
  TeamBar bar;
  int snapshot;
};

// What a team reads throughout; the kernel keeps a copy in shared memory.  WIDE: one
// of the matrices has wide strips (without them the kernels are 2% faster on small
// LPs, whose time is a few chains of instructions an iteration).
template <class T, class M, bool WIDE>
struct TeamData {
  static constexpr bool kWide = WIDE;
  Dev<T> d;
  StripMat<M> A, AT;
  StripMat<double> A64, AT64;
};
template <class D>
__device__ __forceinline__ void team_copy(const D &from, D &to, TeamSmem &sm) {
  static_assert(sizeof(D) % 4 == 0, "copied by words");
  const int *a = reinterpret_cast<const int *>(&from);
  int *b = reinterpret_cast<int *>(&to);
  for (int i = threadIdx.x; i < (int)(sizeof(D) / 4); i += kTeamThreads) b[i] = a[i];
  if (threadIdx.x == 0) sm.target = 0;
  __syncthreads();
}

// Element work in the blocks of a kernel of d.ew_grid blocks (one by one), so
// that its reductions are that kernel's.
template <class Body>
__device__ __forceinline__ void team_blocks(int ew_grid, Body &&body) {
  for (int b = blockIdx.x; b < ew_grid; b += gridDim.x) {
    body(b, b * (long)kThreads + threadIdx.x, (long)ew_grid * kThreads);
    __syncthreads();
  }
}

// KKT evaluation of iteration t; false when a barrier wait ran out.
template <class T, class M, bool WIDE>
__device__ __noinline__ bool team_eval(const TeamData<T, M, WIDE> &sd, const TeamRun r, TeamSmem &sm,
                                       int t, bool infeas, bool restart_check) {
  using Data = TeamData<T, M, WIDE>;
  const Dev<T> &d = sd.d;
  auto on_A = [](const Data &x) -> const auto & { return x.A64; };
  auto on_AT = [](const Data &x) -> const auto & { return x.AT64; };
  if (d.linf) {
    team_phase<2, 1u>(
        sd, on_A, [](const Data &x) { return EvalAEpi<T, double, true, const Dev<T> &>{x.d}; },
        d.p_e1);
    team_phase<3, 1u>(
        sd, on_AT, [](const Data &x) { return EvalATEpi<T, double, true, const Dev<T> &>{x.d}; },
        d.p_e2);
  } else {
    team_phase<2, 0u>(
        sd, on_A, [](const Data &x) { return EvalAEpi<T, double, false, const Dev<T> &>{x.d}; },
        d.p_e1);
    team_phase<3, 0u>(
        sd, on_AT, [](const Data &x) { return EvalATEpi<T, double, false, const Dev<T> &>{x.d}; },
        d.p_e2);
  }
  if (infeas) {
    team_blocks(d.ew_grid, [&](int b, long first, long stride) {
      double a[2] = {0.0, 0.0};
      ray_project(d, first, stride, a);
      block_reduce_fields<2, 3u>(a, sm.red);
      if (threadIdx.x == 0) {
        d.p_i0[b] = a[0];
        d.p_i0[d.ew_grid + b] = a[1];
      }
    });
    if (!team_sync(r.bar, sm)) return false;
    if (blockIdx.x == 0) {
      double v[2];
      block_fold_fields<2, 3u>(d.p_i0, d.ew_grid, sm.red, v);
      if (threadIdx.x == 0) {
        d.ctl->ray_primal_inf_norm = v[0];
        d.ctl->ray_dual_inf_norm = v[1];
      }
    }
    if (!team_sync(r.bar, sm)) return false;
    const T sc = (T)ray_scale(d.ctl);
    team_phase<2, 1u>(
        sd, on_A, [=](const Data &x) { return InfAEpi<T, double, const Dev<T> &>{x.d, sc}; },
        d.p_i1);
    team_phase<3, 2u>(
        sd, on_AT, [=](const Data &x) { return InfATEpi<T, double, const Dev<T> &>{x.d, sc}; },
        d.p_i2);
  }
  if (!team_sync(r.bar, sm)) return false;
  if (blockIdx.x == 0) {
    // the control block in shared memory meanwhile: its fields are read and
    // written one after the other
    __shared__ Ctl ctl;
    static_assert(sizeof(Ctl) % 8 == 0 && sizeof(Ctl) / 8 <= kTeamThreads, "a word a thread");
    double *const local = reinterpret_cast<double *>(&ctl);
    double *const global = reinterpret_cast<double *>(d.ctl);
    if (threadIdx.x < sizeof(Ctl) / 8) local[threadIdx.x] = global[threadIdx.x];
    const EvalSums s = fold_eval(d, infeas, sm.red);
    if (threadIdx.x == 0) eval_scalars(d, &ctl, t, infeas, restart_check, kEvalCheck, s);
    __syncthreads();
    if (threadIdx.x < sizeof(Ctl) / 8) global[threadIdx.x] = local[threadIdx.x];
  }
  return team_sync(r.bar, sm);
}

// Restart of iteration t: the copies and the primal-weight update.
template <class T, class M, bool WIDE>
__device__ __noinline__ bool team_restart(const TeamData<T, M, WIDE> &sd, const TeamRun r, TeamSmem &sm,
                                          int t) {
  const Dev<T> &d = sd.d;
  team_blocks(d.ew_grid, [&](int b, long first, long stride) {
    double a[2] = {0.0, 0.0};
    restart_copy(d, d.x[t & 1], d.y[t & 1], first, stride, a);
    block_reduce_fields<2, 0u>(a, sm.red);
    if (threadIdx.x == 0) {
      d.p_rs[b] = a[0];
      d.p_rs[d.ew_grid + b] = a[1];
    }
  });
  if (!team_sync(r.bar, sm)) return false;
  if (blockIdx.x == 0) {
    double v[2];
    block_fold_fields<2, 0u>(d.p_rs, d.ew_grid, sm.red, v);
    if (threadIdx.x == 0) restart_scalars(d, t, v[0], v[1]);
  }
  return team_sync(r.bar, sm);
}

// An iteration that needs dx, dy and their norms, up to the barrier that ends
// it, and its fixed-point error.
template <class T, class M, bool WIDE>
__device__ __noinline__ bool team_step_fpe(const TeamData<T, M, WIDE> &sd, const TeamRun r, TeamSmem &sm,
                                           T tau, T sigma, T inv_sigma, T w, T omw, int par,
                                           bool major, bool fpe) {
  using Data = TeamData<T, M, WIDE>;
  const Dev<T> &d = sd.d;
  auto on_A = [](const Data &x) -> const auto & { return x.A; };
  auto on_AT = [](const Data &x) -> const auto & { return x.AT; };
  team_phase<1, 0u>(
      sd, on_AT,
      [=](const Data &x) { return TeamPrimal<T, M, true>{x.d, tau, w, omw, par, major}; },
      d.p_pstep);
  if (!team_sync(r.bar, sm)) return false;
  team_phase<1, 0u>(
      sd, on_A,
      [=](const Data &x) {
        return TeamDual<T, M, true>{x.d, sigma, inv_sigma, w, omw, par, major};
      },
      d.p_dstep);
  if (!team_sync(r.bar, sm)) return false;
  if (!fpe) return true;
  team_phase<1, 0u>(
      sd, on_AT, [](const Data &x) { return FpeEpi<T, M, false, const Dev<T> &>{x.d}; }, d.p_fpe);
  if (!team_sync(r.bar, sm)) return false;
  if (blockIdx.x == 0) {
    double pn2, dn2, cross;
    fold_fpe(d, sm.red, pn2, dn2, cross);
    if (threadIdx.x == 0) fpe_scalars(d, pn2, dn2, cross);
  }
  return team_sync(r.bar, sm);
}

__device__ __forceinline__ int ld_flag(const int *p) { return *(const volatile int *)p; }

// What iteration t does (IterFlags) in a byte.
enum TeamFlag {
  kTlEval = 1, kTlInfeas = 2, kTlRestartCheck = 4, kTlMaybeRestart = 8,
  kTlMajor = 16, kTlFpe = 32, kTlFpeRestartOnly = 64, kTlTimed = 128
};
constexpr int kTeamChunk = 1000;  // iterations of a launch

__device__ __forceinline__ bool team_ordinary(const IterFlags &f) {
  return !f.eval && !f.maybe_restart && !f.major_kernel && !f.fpe;
}
static __device__ __noinline__ unsigned team_flags(int t, int F, bool polish) {
  const IterFlags f = iteration_flags(t, F);
  unsigned b = (f.eval ? kTlEval : 0) | (f.infeas && !polish ? kTlInfeas : 0) |
               (f.restart_check ? kTlRestartCheck : 0) | (f.maybe_restart ? kTlMaybeRestart : 0) |
               (f.major_kernel ? kTlMajor : 0) | (f.fpe ? kTlFpe : 0) |
               (f.fpe_restart_only ? kTlFpeRestartOnly : 0);
  // the first ordinary iteration of the second half of each hundred is timed
  if (t % 100 >= 50 && team_ordinary(f)) {
    int u = t - t % 100 + 50;
    while (u < t && !team_ordinary(iteration_flags(u, F))) ++u;
    if (u == t) b |= kTlTimed;
  }
  return b;
}

// Iterations [t0, t1) of the loop (reference src/solver.cu:58-103; at most
// kTeamChunk), up to the one that sets ctl->done.  The order of the parts of
// an iteration, and every scalar decision, are those of
// Solve::enqueue_iteration.  What one iteration hands to the next, other than
// its number, is in shared memory: registers that live across the calls below
// would be spilled, also by the iterations that make none.
template <class T, class M, bool WIDE>
__global__ void __launch_bounds__(kTeamThreads, kTeamCtasPerSm)
    team_loop(const __grid_constant__ TeamData<T, M, WIDE> data, const __grid_constant__ TeamRun run,
              int t0, int t1) {
  using Data = TeamData<T, M, WIDE>;
  __shared__ TeamSmem sm;
  __shared__ Data sd;
  __shared__ TeamRun r;
  __shared__ unsigned char flags[kTeamChunk];
  __shared__ double steps[3];  // tau, sigma, 1 / sigma
  __shared__ int restart_t;
  if (ld_flag(&data.d.ctl->done)) return;  // set by an earlier launch: the same in every CTA
  for (int t = t0 + (int)threadIdx.x; t < t1; t += kTeamThreads)
    flags[t - t0] = (unsigned char)team_flags(t, data.d.F, data.d.polish != 0);
  if (threadIdx.x == 0) {
    r = run;
    const Ctl *c = data.d.ctl;
    steps[0] = c->tau;
    steps[1] = c->sigma;
    steps[2] = c->inv_sigma;
    restart_t = c->restart_t;
  }
  team_copy(data, sd, sm);
  auto on_A = [](const Data &x) -> const auto & { return x.A; };
  auto on_AT = [](const Data &x) -> const auto & { return x.AT; };
  StripHead<M> xT;
  strip_head<false>(sd.AT, team_strip(), xT);
  for (int t = t0; t < t1; ++t) {
    if (flags[t - t0] & kTlEval) {
      const unsigned f = flags[t - t0];
      if (!team_eval(sd, r, sm, t, (f & kTlInfeas) != 0, (f & kTlRestartCheck) != 0)) return;
      if (r.snapshot && ld_flag(&sd.d.ctl->snap_now)) {
        snapshot_copy(sd.d, (long)blockIdx.x * kTeamThreads + threadIdx.x,
                      (long)gridDim.x * kTeamThreads);
        if (!team_sync(r.bar, sm)) return;
      }
      if (ld_flag(&sd.d.ctl->done)) return;
      if ((f & kTlMaybeRestart) && ld_flag(&sd.d.ctl->do_restart)) {
        if (!team_restart(sd, r, sm, t)) return;
        if (threadIdx.x == 0) {
          const volatile Ctl *c = sd.d.ctl;
          steps[0] = c->tau;
          steps[1] = c->sigma;
          steps[2] = c->inv_sigma;
          restart_t = t;
        }
      }
      __syncthreads();
      strip_head<false>(sd.AT, team_strip(), xT);  // again: not kept across the calls
    }
    // Halpern weight (k+1)/(k+2) of the inner iteration k
    const int k = t - restart_t;
    const double wd = k < sd.d.hw_len ? __ldg(sd.d.hw + k) : (double)(k + 1) / (double)(k + 2);
    const int par = t & 1;
    if (flags[t - t0] & kTlFpe) {
      // one that only follows a restart is left out when there was none
      const unsigned f = flags[t - t0];
      if (!team_step_fpe(sd, r, sm, (T)steps[0], (T)steps[1], (T)steps[2], (T)wd,
                                (T)(1.0 - wd), par, (f & kTlMajor) != 0,
                                !(f & kTlFpeRestartOnly) || restart_t == t))
        return;
      strip_head<false>(sd.AT, team_strip(), xT);
      continue;
    }
    const bool major = (flags[t - t0] & kTlMajor) != 0;
    const bool time_it = (flags[t - t0] & kTlTimed) && blockIdx.x == 0 && threadIdx.x == 0;
    const T w = (T)wd, omw = (T)(1.0 - wd);
    unsigned long long tm = 0;
    if (time_it) tm = global_ns();
    {
      const T tau = (T)steps[0];
      team_phase<0, 0u>(
          sd, on_AT,
          [=](const Data &x) { return TeamPrimal<T, M, false>{x.d, tau, w, omw, par, major}; },
          nullptr, xT);
    }
    StripHead<M> xA;
    strip_head<false>(sd.A, team_strip(), xA);
    if (!team_sync(r.bar, sm)) return;
    if (time_it) {
      const unsigned long long now = global_ns();
      sd.d.ctl->live_primal_ns += (double)(now - tm);
      tm = now;
    }
    {
      const T sigma = (T)steps[1], inv_sigma = (T)steps[2];
      team_phase<0, 0u>(
          sd, on_A,
          [=](const Data &x) {
            return TeamDual<T, M, false>{x.d, sigma, inv_sigma, w, omw, par, major};
          },
          nullptr, xA);
    }
    strip_head<false>(sd.AT, team_strip(), xT);
    if (!team_sync(r.bar, sm)) return;
    if (time_it) {
      sd.d.ctl->live_dual_ns += (double)(global_ns() - tm);
      sd.d.ctl->live_n += 1;
    }
  }
}

// The power method by a team (solver.cu); false when it was not launched.
bool launch_team_power(int ctas, cudaStream_t st, const PowDev &d, const StripMat<double> &A,
                       const StripMat<double> &AT, const TeamBar &bar, int maxit);

}  // namespace pdlp
