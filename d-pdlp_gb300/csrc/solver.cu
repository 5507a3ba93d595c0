// solver.cu -- problem upload and the FP64 instantiation of the PDHG solve.
//
// The iteration itself (kernels and the Solve driver) lives in
// solver_impl.cuh; this file holds the pieces defined once: the non-template
// kernels, the host transpose, the device-resident problem, and
// Solve<double, double>.
#include <string.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <exception>
#include <mutex>
#include <future>
#include <thread>

#include "solver_impl.cuh"

namespace pdlp {

__global__ void k_set_tbase(Ctl *ctl, int t) { ctl->t_base = t; }
__global__ void k_loop_start(Ctl *ctl) { ctl->t_start_ns = global_ns(); }
__global__ void k_set_steps(Ctl *c) { set_steps(c); }
// Halpern weights (k+1)/(k+2), the quotients the iteration would form
__global__ void k_halpern_table(double *hw, int len) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < len) hw[k] = (double)(k + 1) / (double)(k + 2);
}

// ---- power method element kernels (utils.cu:107-153), FP64
__global__ void __launch_bounds__(kThreads) k_pm_norm(PowDev d, const double *v) {
  if (d.ctl->pm_done) return;
  __shared__ double red[16];
  double a[1] = {0.0};
  long stride = (long)gridDim.x * kThreads;
  for (long i = blockIdx.x * (long)kThreads + threadIdx.x; i < d.m; i += stride)
    a[0] += v[i] * v[i];
  block_reduce_fields<1, 0u>(a, red);
  if (threadIdx.x == 0) d.p_pr[blockIdx.x] = a[0];
}

__global__ void __launch_bounds__(kThreads) k_pm_norm_fin(PowDev d) {
  if (d.ctl->pm_done) return;
  __shared__ double sm[32];
  double s = block_fold<false>(d.p_pr, d.ew_grid, sm);
  if (threadIdx.x == 0) d.ctl->pm_inv_norm = 1.0 / sqrt(s);
}

__global__ void __launch_bounds__(kThreads) k_pm_dot_fin(PowDev d) {
  Ctl *c = d.ctl;
  if (c->pm_done) return;
  __shared__ double sm[32];
  double v[2];  // q.v', |v'|^2
  fold_site<2, 0u>(d.p_pa, d.nblkA, d.lp_pa, d.nlongA, sm, v);
  if (threadIdx.x == 0) {
    c->pm_sigma_sq = v[0];
    c->pm_res = v[1];  // |v'|^2, turned into 1/|v'| after the residual
  }
}

// block `b` of d.ew_grid: its partial of |v' - sigma^2 q|^2
__device__ __forceinline__ void resid_block(const PowDev &d, const double *v, const double *vnext,
                                            double inv, double ns, int b, double *red) {
  double a[1] = {0.0};
  const long stride = (long)d.ew_grid * kThreads;
#pragma unroll 2
  for (long i = b * (long)kThreads + threadIdx.x; i < d.m; i += stride) {
    double q = inv * v[i];
    double r = 1.0 * vnext[i] + ns * q;
    a[0] += r * r;
  }
  block_reduce_fields<1, 0u>(a, red);
  if (threadIdx.x == 0) d.p_pr[b] = a[0];
}
__global__ void __launch_bounds__(kThreads)
    k_pm_resid(PowDev d, const double *v, const double *vnext) {
  if (d.ctl->pm_done) return;
  __shared__ double red[16];
  resid_block(d, v, vnext, d.ctl->pm_inv_norm, -d.ctl->pm_sigma_sq, blockIdx.x, red);
}

__global__ void __launch_bounds__(kThreads) k_pm_resid_fin(PowDev d) {
  Ctl *c = d.ctl;
  if (c->pm_done) return;
  __shared__ double sm[32];
  double s = block_fold<false>(d.p_pr, d.ew_grid, sm);
  if (threadIdx.x == 0) {
    c->pm_iters++;
    double res = sqrt(s);
    c->pm_inv_norm = 1.0 / sqrt(c->pm_res);
    c->pm_res = res;
    if (res < d.sv_tol) {
      c->pm_done = 1;
      __threadfence_system();
      d.hflag->pm_done = 1;
    }
  }
}

// ---- strip format
__global__ void k_invert(int n, const int *__restrict__ perm, int *__restrict__ inv) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    inv[perm[i]] = (int)i;
}
// dst[i] = src[perm[i]] (null perm: src[i]) for several vectors, one to a grid row
struct GatherList {
  const double *src[7];
  double *dst[7];
  const int *perm[7];
  int count[7];
};
__global__ void k_gather(const __grid_constant__ GatherList g) {
  const int v = blockIdx.y;
  const double *src = g.src[v];
  const int *perm = g.perm[v];
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < g.count[v];
       i += (long)gridDim.x * blockDim.x)
    g.dst[v][i] = src[perm ? perm[i] : i];
}
__global__ void k_gather_bytes(int n, const unsigned char *__restrict__ src,
                               const int *__restrict__ perm, unsigned char *__restrict__ dst) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[i] = src[perm[i]];
}
__global__ void k_scatter_back(int n, const double *__restrict__ src, const int *__restrict__ perm,
                               double *__restrict__ dst) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    dst[perm[i]] = src[i];
}
void launch_gather(int n, const double *src, const int *perm, double *dst, cudaStream_t st) {
  if (n <= 0) return;
  k_gather<<<grid_for(n), kThreads, 0, st>>>(GatherList{{src}, {dst}, {perm}, {n}});
  PDLP_LAUNCH_CHECK();
}
void launch_scatter(int n, const double *src, const int *perm, double *dst, cudaStream_t st) {
  if (n <= 0) return;
  k_scatter_back<<<grid_for(n), kThreads, 0, st>>>(n, src, perm, dst);
  PDLP_LAUNCH_CHECK();
}

// The stored elements of a strip-format matrix from entries scol / sval in rows
// sptr: row i is the source's row perm[i] with its entries in their order, whose
// k-th is entry k or pos[k]; column j becomes icol[j] (null perm, pos, icol: the
// identity).  A warp per front item, then a warp per strip.
__global__ void __launch_bounds__(kThreads)
    k_strip_fill(StripMat<double> A, const int *__restrict__ sptr, const int *__restrict__ scol,
                 const double *__restrict__ sval, const int *__restrict__ pos,
                 const int *__restrict__ perm, const int *__restrict__ icol,
                 int *__restrict__ col, double *__restrict__ val) {
  const int lane = threadIdx.x & 31;
  const int W = gridDim.x * (kThreads / 32);
  auto take = [&](int k, int &c, double &v) {
    const int q = pos ? pos[k] : k;
    c = scol[q];
    if (icol) c = icol[c];
    v = sval[q];
  };
  for (int w = (blockIdx.x * kThreads + threadIdx.x) >> 5; w < A.p.nitem + A.p.nstrip; w += W) {
    if (w < A.p.nitem) {
      const int4 b = A.p.item[w];
      const int rows = b.y < 0 ? 1 : b.y, step = b.y < 0 ? 256 : 32;
      for (int i = b.x; i < b.x + rows; ++i) {
        const int from = sptr[perm ? perm[i] : i] - A.ptr[i];  // source less place
        const int first = b.y < 0 ? b.z : A.ptr[i], end = b.y < 0 ? b.w : A.ptr[i + 1];
        for (int k = first + lane; k < end; k += step) take(from + k, col[k], val[k]);
      }
      continue;
    }
    const int s = w - A.p.nitem;
    const StripPlace place = strip_place(A.p, A.rows, s);
    const int lg = place.lg, row = place.row + (lane >> lg), sub = lane & ((1 << lg) - 1);
    int a = 0, len = 0;
    if (row < place.end) {
      const int r = perm ? perm[row] : row;
      a = sptr[r];
      len = sptr[r + 1] - a;
    }
    const size_t o0 = (size_t)A.p.off[s] * 32 + lane;
    const int width = A.p.off[s + 1] - A.p.off[s];
    for (int k = 0; k < width; ++k) {
      int c = -1;
      double v = 0.0;
      const int e = (k << lg) + sub;
      if (e < len) take(a + e, c, v);
      col[o0 + (size_t)k * 32] = c;
      val[o0 + (size_t)k * 32] = v;
    }
  }
}

template <bool WIDE>
struct TeamPower {
  static constexpr bool kWide = WIDE;
  PowDev d;
  StripMat<double> A, AT;
};

// The power method (reference src/utils.cu:66-171): iterations until the
// residual is below sv_tol or `maxit` are done, two barriers each.  Every CTA
// folds the sums itself; the residual of an iteration is checked after the
// next one's A^T product, which writes nothing the result depends on.
template <bool WIDE>
__global__ void __launch_bounds__(kTeamThreads, kTeamCtasPerSm)
    team_power(const __grid_constant__ TeamPower<WIDE> data, const __grid_constant__ TeamBar bar,
               int maxit) {
  __shared__ TeamSmem sm;
  __shared__ TeamPower<WIDE> sd;
  Ctl *c = data.d.ctl;
  if (ld_flag(&c->pm_done)) return;
  team_copy(data, sd, sm);
  const PowDev &d = sd.d;
  int it = 0;
  double inv = c->pm_inv_norm, sigma_sq = 0.0, res = 0.0;
  bool check = false;  // the last iteration left partial sums of its residual
  StripHead<double> xT;
  strip_head<false>(sd.AT, team_strip(), xT);
  for (;;) {
    if (it < maxit)
      team_phase<0, 0u>(
          sd, [](const TeamPower<WIDE> &x) -> const auto & { return x.AT; },
          [=](const TeamPower<WIDE> &x) {
            return PowAtEpi<const PowDev &>{x.d, (it & 1) ? x.d.v[1] : x.d.v[0], inv};
          },
          nullptr, xT);
    StripHead<double> xA;
    strip_head<false>(sd.A, team_strip(), xA);
    if (!team_sync(bar, sm)) return;
    if (check) {  // residual of iteration it - 1
      double v[1];
      block_fold_fields<1, 0u>(d.p_pr, d.ew_grid, sm.red, v);
      res = sqrt(v[0]);
    }
    // `>=`: a limit below zero ends it here too (a launch must always end)
    if (it >= maxit || (check && res < d.sv_tol)) break;
    team_phase<2, 0u>(
        sd, [](const TeamPower<WIDE> &x) -> const auto & { return x.A; },
        [=](const TeamPower<WIDE> &x) {
          return PowAEpi<const PowDev &>{x.d, (it & 1) ? x.d.v[1] : x.d.v[0],
                                         (it & 1) ? x.d.v[0] : x.d.v[1], inv};
        },
        d.p_pa, xA);
    strip_head<false>(sd.AT, team_strip(), xT);
    if (!team_sync(bar, sm)) return;
    double v[2];  // q.v', |v'|^2
    fold_site<2, 0u>(d.p_pa, d.nblkA, d.lp_pa, d.nlongA, sm.red, v);
    sigma_sq = v[0];
    // |v' - sigma^2 q|^2 = |v'|^2 - sigma^4, up to rounding of about 1e-15
    // |v'|^2: the residual itself is only summed where that does not already
    // show that it is far above the tolerance
    const double about = v[1] - sigma_sq * sigma_sq;
    check = !(about - 1e-12 * v[1] > 4.0 * d.sv_tol * d.sv_tol) || it + 1 == maxit;
    if (check)
      for (int b = blockIdx.x; b < d.ew_grid; b += gridDim.x) {
        resid_block(d, (it & 1) ? d.v[1] : d.v[0], (it & 1) ? d.v[0] : d.v[1], inv, -sigma_sq, b,
                    sm.red);
        __syncthreads();
      }
    inv = 1.0 / sqrt(v[1]);
    ++it;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    c->pm_iters = it;
    c->pm_sigma_sq = sigma_sq;
    c->pm_inv_norm = inv;
    c->pm_res = res;
    c->pm_done = check && res < d.sv_tol ? 1 : 0;
    if (c->pm_done) {
      __threadfence_system();
      d.hflag->pm_done = 1;
    }
  }
}

bool launch_team_power(int ctas, cudaStream_t st, const PowDev &d, const StripMat<double> &A,
                       const StripMat<double> &AT, const TeamBar &bar, int maxit) {
  return A.p.nwide + AT.p.nwide > 0
             ? team_launch(ctas, team_power<true>, st, TeamPower<true>{d, A, AT}, bar, maxit)
             : team_launch(ctas, team_power<false>, st, TeamPower<false>{d, A, AT}, bar, maxit);
}

void team_reset(unsigned *count, cudaStream_t st) {
  const char *e = getenv("PDLP_TEAM_FAIL");
  // 0xC0C0C0C0 arrivals are 1.06e9 short of 0
  PDLP_CUDA(cudaMemsetAsync(count, e && e[0] == '1' ? 0xC0 : 0, sizeof(unsigned), st));
}

namespace {
std::atomic<int> g_solves{0};
std::mutex g_team_mu;
}  // namespace

SolveInFlight::SolveInFlight() { g_solves.fetch_add(1); }
SolveInFlight::~SolveInFlight() { g_solves.fetch_sub(1); }
TeamTurn::TeamTurn(bool wanted) {
  held_ = wanted && alone() && g_team_mu.try_lock();
}
TeamTurn::~TeamTurn() {
  if (held_) g_team_mu.unlock();
}
bool TeamTurn::alone() { return g_solves.load() <= 1; }

// A^T in CSR, entries of each column in row order (a stable counting sort).
// Matrices of 4M+ non-zeros are transposed by up to 8 threads, each owning a
// range of columns (balanced by non-zeros) and scanning every row in order,
// so the result is the serial one, bit for bit.
void host_transpose(int m, int n, const int *ap, const int *aj, const double *ax,
                    std::vector<int> &tp, host_buf<int> &tj, host_buf<double> &tx) {
  const int nnz = ap[m];
  tp.assign((size_t)n + 1, 0);
  tj.resize(nnz);
  tx.resize(nnz);
  const unsigned hw = std::thread::hardware_concurrency();
  const int T = nnz >= 4000000 && n > 0 ? (int)std::min(8u, hw ? hw : 1u) : 1;
  auto run = [&](auto &&f) {
    std::vector<std::thread> th;
    for (int t = 1; t < T; ++t) th.emplace_back(f, t);
    f(0);
    for (auto &x : th) x.join();
  };
  // column counts: thread t owns columns [n t / T, n (t+1) / T)
  run([&](int t) {
    const int c0 = (int)((long)n * t / T), c1 = (int)((long)n * (t + 1) / T);
    for (int k = 0; k < nnz; ++k) {
      const int c = aj[k];
      if (c >= c0 && c < c1) tp[c + 1]++;
    }
  });
  for (int c = 0; c < n; ++c) tp[c + 1] += tp[c];
  // scatter: column ranges of about nnz / T entries each
  std::vector<int> cut(T + 1, n);
  cut[0] = 0;
  for (int t = 1; t < T; ++t)
    cut[t] = std::max(cut[t - 1], (int)(std::lower_bound(tp.begin(), tp.end(),
                                                         (int)((long)nnz * t / T)) - tp.begin()));
  cut[T] = n;
  run([&](int t) {
    const int c0 = std::min(cut[t], n), c1 = std::min(cut[t + 1], n);
    if (c0 >= c1) return;
    std::vector<int> next(tp.begin() + c0, tp.begin() + c1);
    for (int r = 0; r < m; ++r)
      for (int k = ap[r]; k < ap[r + 1]; ++k) {
        const int c = aj[k];
        if (c >= c0 && c < c1) {
          const int pos = next[c - c0]++;
          tj[pos] = r;
          tx[pos] = ax[k];
        }
      }
  });
}

// Non-zeros per thread-block tile.  PDLP_SPMV_TILE (512, 1024 or 2048)
// overrides the size rule (1024 measured fastest on the 20M-nnz power-law and
// transport LPs at 6 resident blocks per SM).
static int pick_tile(long nnz) {
  if (const char *e = getenv("PDLP_SPMV_TILE")) {
    int t = atoi(e);
    if (t == 512 || t == 1024 || t == 2048) return t;
  }
  return nnz >= 2000000 ? 1024 : 512;
}

// Non-zeros per block of a row longer than a tile: 8192 (at most 8 tiles).
// Long chunks amortise the block's FP64 reduction, barriers and ticket over
// more non-zeros (measured on the 20M-nnz LPs: power-law primal step -12%,
// transport dual step -25% against one tile per chunk; 16384 loses to load
// imbalance).  PDLP_SPMV_CHUNK (a multiple of the tile, at most 16384)
// overrides the default.
static int pick_chunk(int tile) {
  if (const char *e = getenv("PDLP_SPMV_CHUNK")) {
    int c = atoi(e);
    if (c >= tile && c <= 16384 && c % tile == 0) return c;
  }
  return tile * 8 < 8192 ? tile * 8 : 8192;
}

int kernel_override() {
  static const int v = [] {
    const char *e = getenv("PDLP_STEP_KERNEL");
    if (e && strcmp(e, "pipe") == 0) return 1;
    if (e && strcmp(e, "fused") == 0) return 0;
    return -1;
  }();
  return v;
}

namespace {
// Host threads for the upload's passes over the non-zeros (LPs of 2M+
// non-zeros; smaller ones stay on the calling thread).
int upload_threads(long nnz) {
  const unsigned hw = std::thread::hardware_concurrency();
  return nnz >= (1L << 21) ? (int)std::min(16u, hw ? hw : 1u) : 1;
}

// f(begin, end) over [0, count) in T contiguous slices, slice 0 on this thread
template <class F>
void parallel_slices(int T, long count, F &&f) {
  if (T <= 1) {
    f(0L, count);
    return;
  }
  std::vector<std::thread> th;
  for (int t = 1; t < T; ++t) th.emplace_back([&f, t, T, count] { f(count * t / T, count * (t + 1) / T); });
  f(0L, count / T);
  for (auto &x : th) x.join();
}
}  // namespace

DevProblem::~DevProblem() {
  if (!arena) return;  // a view of another problem
  if (fp32 && fp32->mem) dev_free(fp32->mem, owner);
  dev_free(arena, owner);
}

namespace {
// The rows' FP32 sums of A and A^T (strip.cuh) in their original order.
struct Fp32Host {
  std::vector<unsigned char> A, AT;
  bool pairs_A = false, pairs_AT = false;
};
Fp32Host fp32_order_host(int m, int n, const int *ptr, const int *tptr, int tile, int threads) {
  Fp32Host h;
  auto one = [&](int rows, const int *p, int nv, std::vector<unsigned char> &sums, bool &pairs) {
    pairs = strip_pairs(rows, p);
    if (pairs) strip_sums_pipe(rows, p, nv, sums);
    else strip_sums_fused(rows, p, tile, pick_chunk(tile), sums);
  };
  auto of_A = [&] { one(m, ptr, 4, h.A, h.pairs_A); };
  std::future<void> other;
  if (threads > 1) other = std::async(std::launch::async, of_A);
  else of_A();
  one(n, tptr, 5, h.AT, h.pairs_AT);
  if (other.valid()) other.get();
  return h;
}
// ... and on the device in the format's order.
void fp32_order_upload(const DevProblem &P, const Fp32Host &h, Fp32Order &o, cudaStream_t st) {
  const size_t vm = P.m, vn = P.n;
  Sizer z;
  z.add<unsigned char>(vm);
  z.add<unsigned char>(vn);
  o.mem = dev_alloc(z.bytes, st);
  struct Scratch {
    void *p;
    cudaStream_t st;
    ~Scratch() { dev_free(p, st); }
  } raw{dev_alloc(std::max(vm, vn), st), st};
  Arena ar{(char *)o.mem, 0};
  auto put = [&](const std::vector<unsigned char> &v, const int *perm, const unsigned char *&out) {
    unsigned char *dst = ar.take<unsigned char>(v.size());
    out = dst;
    if (v.empty()) return;
    PDLP_CUDA(cudaMemcpyAsync(perm ? raw.p : dst, v.data(), v.size(), cudaMemcpyHostToDevice, st));
    if (!perm) return;
    k_gather_bytes<<<grid_for((long)v.size()), kThreads, 0, st>>>(
        (int)v.size(), (const unsigned char *)raw.p, perm, dst);
    PDLP_LAUNCH_CHECK();
  };
  put(h.A, P.perm_m, o.A);
  put(h.AT, P.perm_n, o.AT);
  o.pairs_A = h.pairs_A;
  o.pairs_AT = h.pairs_AT;
  PDLP_CUDA(cudaStreamSynchronize(st));  // also for solves on other streams
  o.made = true;
}
}  // namespace

const Fp32Order &DevProblem::fp32_order(cudaStream_t st) const {
  Fp32Order &o = *fp32;
  std::lock_guard<std::mutex> lk(o.mu);
  if (!o.made) {
    if (o.mem) dev_free(o.mem, st);  // of an attempt that failed
    o.mem = nullptr;
    fp32_order_upload(*this, fp32_order_host(m, n, o.ptr.data(), o.tptr.data(), tile,
                                             upload_threads(nnz)), o, st);
    o.ptr = {};
    o.tptr = {};
  }
  return o;
}

DevProblem *upload_problem(const lp_problem_t *prob, cudaStream_t st, int kernel,
                           bool for_fp32) {
  const int n = prob->num_variables, m = prob->num_constraints;
  const int nnz = prob->constraint_matrix_num_nonzeros;
  // A malformed CSR must never reach the host transpose or a device gather.
  {
    const int *rp = prob->constraint_matrix_row_pointers;
    const int *cj = prob->constraint_matrix_col_indices;
    bool ok = n >= 0 && m >= 0 && nnz >= 0 && rp &&
              (nnz == 0 || (cj && prob->constraint_matrix_values)) &&
              (n == 0 || (prob->objective_vector && prob->variable_lower_bound &&
                          prob->variable_upper_bound)) &&
              (m == 0 || (prob->constraint_lower_bound && prob->constraint_upper_bound));
    if (ok) ok = rp[0] == 0 && rp[m] == nnz;
    for (int r = 0; ok && r < m; ++r) ok = rp[r] <= rp[r + 1];
    if (ok) {
      std::atomic<bool> bad{false};
      parallel_slices(upload_threads(nnz), nnz, [&](long a, long b) {
        for (long k = a; k < b; ++k)
          if (cj[k] < 0 || cj[k] >= n) {
            bad.store(true, std::memory_order_relaxed);
            return;
          }
      });
      ok = !bad.load();
    }
    if (!ok) throw std::runtime_error("invalid CSR matrix (row pointers or column indices)");
  }
  auto P = std::make_unique<DevProblem>();
  P->owner = st;
  P->m = m;
  P->n = n;
  P->nnz = nnz;
  P->tile = pick_tile(nnz);
  P->c0 = prob->objective_constant;
  // row pointers of A^T (column counts of A, prefix-summed) for the plans;
  // A^T itself is built on the device after A is uploaded
  std::vector<int> tp((size_t)n + 1, 0);
  {
    const int *cj = prob->constraint_matrix_col_indices;
    int *cnt = tp.data() + 1;
    const int T = upload_threads(nnz);
    if (T > 1) {
      parallel_slices(T, nnz, [&](long a, long b) {
        for (long k = a; k < b; ++k) __atomic_fetch_add(cnt + cj[k], 1, __ATOMIC_RELAXED);
      });
    } else {
      for (int k = 0; k < nnz; ++k) cnt[cj[k]]++;
    }
    for (int c = 0; c < n; ++c) tp[c + 1] += tp[c];
  }
  const bool strips = kernel < 0;  // else that kernel's CSR
  P->kernel = kernel;
  P->strips = strips;
  int dev = 0, nsm = kNumSms;
  PDLP_CUDA(cudaGetDevice(&dev));
  PDLP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  P->nsm = nsm;
  std::vector<int4> blkA, blkT;
  std::vector<int2> lrA, lrT;
  const int chunk = pick_chunk(P->tile);
  // pipelined step kernel: the dual step (A) stages 4 row vectors, the
  // primal step (A^T) 5.  A's plans are built on a second thread for large
  // LPs, beside A^T's.
  std::vector<int4> pblkA, pblkT;
  std::vector<int2> plrA, plrT;
  StripHost shA, shT;
  std::future<Fp32Host> fp32_host;
  if (strips && for_fp32)
    fp32_host = std::async(upload_threads(nnz) > 1 ? std::launch::async : std::launch::deferred,
                           [&] {
                             return fp32_order_host(m, n, prob->constraint_matrix_row_pointers,
                                                    tp.data(), P->tile, upload_threads(nnz));
                           });
  auto plans_A = [&] {
    if (strips) {
      build_strip_host(m, prob->constraint_matrix_row_pointers, nsm, P->tile, chunk, shA);
      return;
    }
    build_plan_host(m, prob->constraint_matrix_row_pointers, P->tile, blkA, lrA, chunk);
    build_pipe_plan_host(m, prob->constraint_matrix_row_pointers, 4, pblkA, plrA);
  };
  std::exception_ptr failed_A;
  std::thread thread_A;
  if (upload_threads(nnz) > 1)
    thread_A = std::thread([&] {
      try {
        plans_A();
      } catch (...) {
        failed_A = std::current_exception();
      }
    });
  else
    plans_A();
  try {
    if (strips) {
      build_strip_host(n, tp.data(), nsm, P->tile, chunk, shT);
    } else {
      build_plan_host(n, tp.data(), P->tile, blkT, lrT, chunk);
      build_pipe_plan_host(n, tp.data(), 5, pblkT, plrT);
    }
  } catch (...) {
    if (thread_A.joinable()) thread_A.join();
    throw;
  }
  if (thread_A.joinable()) thread_A.join();
  if (failed_A) std::rethrow_exception(failed_A);
  // norms of the unscaled objective and bounds (reference pdlp_core_op.cu:232-286)
  {
    double ss = 0, mx = 0;
    for (int i = 0; i < n; ++i) {
      double v = prob->objective_vector[i];
      mx = fmax(mx, fabs(v));
      ss += v * v;
    }
    P->cnorm_l2 = sqrt(ss);
    P->cnorm_linf = mx;
    ss = 0;
    mx = 0;
    for (int i = 0; i < m; ++i) {
      double lo = prob->constraint_lower_bound[i], up = prob->constraint_upper_bound[i];
      if (isfinite(lo) && lo != up) {
        mx = fmax(mx, fabs(lo));
        ss += lo * lo;
      }
      if (isfinite(up)) {
        mx = fmax(mx, fabs(up));
        ss += up * up;
      }
    }
    P->bnorm_l2 = sqrt(ss);
    P->bnorm_linf = mx;
  }
  const size_t vn = n, vm = m;
  Sizer z;
  if (strips) {
    for (const StripHost *h : {&shA, &shT}) {
      z.add<int>(h->fptr.size()); z.add<int>(h->off.size());
      z.add<int4>(h->item.size()); z.add<int2>(h->lrow.size());
      z.add<int>(h->perm.size());
      z.add<int>(h->store); z.add<double>(h->store);
    }
  } else {
    z.add<int>(vm + 1); z.add<int>(nnz); z.add<double>(nnz);
    z.add<int>(vn + 1); z.add<int>(nnz); z.add<double>(nnz);
  }
  z.add<int4>(blkA.size()); z.add<int2>(lrA.size());
  z.add<int4>(blkT.size()); z.add<int2>(lrT.size());
  z.add<int4>(pblkA.size()); z.add<int2>(plrA.size());
  z.add<int4>(pblkT.size()); z.add<int2>(plrT.size());
  for (int i = 0; i < 3; ++i) z.add<double>(vn);
  for (int i = 0; i < 2; ++i) z.add<double>(vm);
  if (prob->primal_start) z.add<double>(vn);
  if (prob->dual_start) z.add<double>(vm);
  P->arena = dev_alloc(z.bytes, st);
  P->bytes = z.bytes;
  Arena ar{(char *)P->arena, 0};
  auto mat = [&](DevCsr &M, int rows, int cols, std::vector<int4> &blk, std::vector<int2> &lr,
                 std::vector<int4> &pblk, std::vector<int2> &plr) {
    M.rows = rows;
    M.cols = cols;
    M.nnz = nnz;
    M.ptr = ar.take<int>((size_t)rows + 1);
    M.col = ar.take<int>(nnz);
    M.val = ar.take<double>(nnz);
    M.plan.rows = rows;
    M.plan.nblk = (int)blk.size();
    M.plan.nlong = (int)lr.size();
    M.plan.tile = P->tile;
    // register-path kernel variant for matrices of short rows of 16+ non-zeros
    // (tiles of 1024 only); PDLP_SPMV_DIRECT=0/1 overrides the rule
    M.plan.direct = P->tile == 1024 && plan_direct(blk, nnz);
    if (const char *e = getenv("PDLP_SPMV_DIRECT")) M.plan.direct = P->tile == 1024 && atoi(e) != 0;
    M.plan.blk = ar.take<int4>(blk.size());
    M.plan.lrow = ar.take<int2>(lr.size());
    if (!blk.empty())
      PDLP_CUDA(cudaMemcpyAsync(M.plan.blk, blk.data(), blk.size() * 16, cudaMemcpyHostToDevice, st));
    if (!lr.empty())
      PDLP_CUDA(cudaMemcpyAsync(M.plan.lrow, lr.data(), lr.size() * 8, cudaMemcpyHostToDevice, st));
    M.pipe.ntile = (int)pblk.size();
    M.pipe.nlong = (int)plr.size();
    const long cap = (long)nsm * kPipeCtasPerSm;
    M.pipe.grid = (int)(M.pipe.ntile < cap ? M.pipe.ntile : cap);
    M.pipe.blk = ar.take<int4>(pblk.size());
    M.pipe.lrow = ar.take<int2>(plr.size());
    if (!pblk.empty())
      PDLP_CUDA(cudaMemcpyAsync(M.pipe.blk, pblk.data(), pblk.size() * 16, cudaMemcpyHostToDevice, st));
    if (!plr.empty())
      PDLP_CUDA(cudaMemcpyAsync(M.pipe.lrow, plr.data(), plr.size() * 8, cudaMemcpyHostToDevice, st));
  };
  // Host arrays on their way to consecutive places on the device.  Up to
  // kPackBytes they go in one copy from one buffer: a small LP's upload is the
  // number of its copies (20,000 non-zeros: 0.32 ms with 19 of them, 0.23 before
  // there were strips).
  constexpr size_t kPackBytes = 1 << 20;
  struct Sending {
    std::vector<std::array<const void *, 2>> at;  // source, place
    std::vector<size_t> bytes;
    std::vector<char> packed;
    void add(void *dst, const void *src, size_t b) {
      if (b == 0) return;
      at.push_back({src, dst});
      bytes.push_back(b);
    }
    void go(cudaStream_t st) {
      if (at.empty()) return;
      char *const base = (char *)at[0][1];
      const size_t all = (const char *)at.back()[1] + bytes.back() - base;
      if (all <= kPackBytes) {
        packed.resize(all);
        for (size_t i = 0; i < at.size(); ++i)
          memcpy(packed.data() + ((const char *)at[i][1] - base), at[i][0], bytes[i]);
        PDLP_CUDA(cudaMemcpyAsync(base, packed.data(), all, cudaMemcpyHostToDevice, st));
        return;
      }
      for (size_t i = 0; i < at.size(); ++i)
        PDLP_CUDA(cudaMemcpyAsync((void *)at[i][1], at[i][0], bytes[i], cudaMemcpyHostToDevice, st));
    }
  };
  Sending index, input;
  auto up = [&](auto *&dst, const auto &src) {
    using E = typename std::remove_reference_t<decltype(src)>::value_type;
    E *p = ar.take<E>(src.size());
    dst = p;
    index.add(p, src.data(), src.size() * sizeof(E));
  };
  auto strip = [&](DevCsr &M, int rows, int cols, const StripHost &h, const int *&perm) {
    M.rows = rows;
    M.cols = cols;
    M.nnz = nnz;
    StripPlan &p = M.strip;
    p.on = 1;
    p.nfront = (int)h.fptr.size() - 1;
    p.nitem = (int)h.item.size();
    p.nlong = (int)h.lrow.size();
    p.nstrip = (int)h.off.size() - 1;
    p.nwide = h.nwide;
    p.wide_end = h.wide_end;
    p.lg = h.lg;
    p.lgw = h.lgw;
    p.store = h.store;
    // (rows stand in decreasing length: the first strip is the widest)
    p.narrow = p.nitem == 0 && p.nwide == 0 && p.lg == 0 && p.nstrip > 0 &&
               h.off[1] - h.off[0] <= kNarrow;
    const long warps = (long)p.nitem + p.nstrip, per = kThreads / 32;
    p.grid = (int)((warps + per - 1) / per);
    up(M.ptr, h.fptr);
    up(p.off, h.off);
    up(p.item, h.item);
    up(p.lrow, h.lrow);
    if (!h.perm.empty()) up(perm, h.perm);
  };
  if (strips) {
    strip(P->A, m, n, shA, P->perm_m);
    strip(P->AT, n, m, shT, P->perm_n);
    for (DevCsr *M : {&P->A, &P->AT}) {
      M->col = ar.take<int>(M->strip.store);
      M->val = ar.take<double>(M->strip.store);
    }
    P->A.strip.unit_parts = P->AT.strip.unit_parts =
        team_ctas(nnz, P->A.strip, P->AT.strip, nsm) > 0;
    index.go(st);
  } else {
    mat(P->A, m, n, blkA, lrA, pblkA, plrA);
    mat(P->AT, n, m, blkT, lrT, pblkT, plrT);
  }
  P->c = ar.take<double>(vn);
  P->lv = ar.take<double>(vn);
  P->uv = ar.take<double>(vn);
  P->lc = ar.take<double>(vm);
  P->uc = ar.take<double>(vm);
  if (prob->primal_start) P->xs = ar.take<double>(vn);
  if (prob->dual_start) P->ys = ar.take<double>(vm);
  struct Vec {
    double *dst;
    const double *src;
    size_t count;
    const int *perm;
  };
  std::vector<Vec> vecs = {{P->c, prob->objective_vector, vn, P->perm_n},
                           {P->lv, prob->variable_lower_bound, vn, P->perm_n},
                           {P->uv, prob->variable_upper_bound, vn, P->perm_n},
                           {P->lc, prob->constraint_lower_bound, vm, P->perm_m},
                           {P->uc, prob->constraint_upper_bound, vm, P->perm_m}};
  if (P->xs) vecs.push_back({P->xs, prob->primal_start, vn, P->perm_n});
  if (P->ys) vecs.push_back({P->ys, prob->dual_start, vm, P->perm_m});
  auto direct = [&](const Vec &v) { return !v.perm && v.count * 8 > kPackBytes; };
  // device scratch of the upload, released on its stream: A as given, what its
  // stable transpose (reference: cusparseCsr2cscEx2, src/pdlp_core_op.cu:109-130)
  // needs beside the places of the strips, and the vectors as given
  struct Scratch {
    void *p;
    cudaStream_t st;
    ~Scratch() { dev_free(p, st); }
  };
  Sizer zs;
  if (strips) {
    zs.add<int>(vm + 1); zs.add<int>(nnz); zs.add<double>(nnz);
    for (const Vec &v : vecs)
      if (!direct(v)) zs.add<double>(v.count);
    zs.add<int>(vn + 1); zs.add<int>(vm); zs.add<int>(vn);
    zs.add<char>(column_sort_hist_bytes(nnz));
  } else {
    zs.add<char>(device_transpose_scratch_bytes(n, nnz));
  }
  const Scratch scratch{dev_alloc(zs.bytes, st), st};
  Arena sa{(char *)scratch.p, 0};
  if (strips) {
    int *const ptr = sa.take<int>(vm + 1), *const col = sa.take<int>(nnz);
    double *const val = sa.take<double>(nnz);
    input.add(ptr, prob->constraint_matrix_row_pointers, (vm + 1) * 4);
    input.add(col, prob->constraint_matrix_col_indices, (size_t)nnz * 4);
    input.add(val, prob->constraint_matrix_values, (size_t)nnz * 8);
    GatherList list{};
    int lists = 0;
    size_t most = 0;
    for (const Vec &v : vecs) {
      if (direct(v)) {
        PDLP_CUDA(cudaMemcpyAsync(v.dst, v.src, v.count * 8, cudaMemcpyHostToDevice, st));
        continue;
      }
      double *const raw = sa.take<double>(v.count);
      input.add(raw, v.src, v.count * 8);
      list.src[lists] = raw;
      list.dst[lists] = v.dst;
      list.perm[lists] = v.perm;
      list.count[lists++] = (int)v.count;
      most = std::max(most, v.count);
    }
    input.go(st);
    int *const tptr = sa.take<int>(vn + 1);
    int *const inv_m = sa.take<int>(vm), *const inv_n = sa.take<int>(vn);
    int *const hist = (int *)sa.take<char>(column_sort_hist_bytes(nnz));
    // the sort's arrays are where the strips will be: its result (positions and
    // rows) in A's place, which is filled last, its keys in A^T's
    int *const inA = P->A.col, *const inT = P->AT.col;
    const size_t nz = nnz;
    const ColumnSort sort{inT, inT + nz, inA, inA + nz, inA + 2 * nz, hist};
    const int *const pos = device_column_sort(m, n, nnz, ptr, col, sort, tptr, st);
    if (P->perm_m) k_invert<<<grid_for(m), kThreads, 0, st>>>(m, P->perm_m, inv_m);
    if (P->perm_n) k_invert<<<grid_for(n), kThreads, 0, st>>>(n, P->perm_n, inv_n);
    auto fill = [&](DevCsr &M, const int *sp, const int *sc, const double *sv, const int *at,
                    const int *perm, const int *icol) {
      const long warps = (long)M.strip.nitem + M.strip.nstrip;
      if (warps == 0) return;
      k_strip_fill<<<grid_for(warps * 32), kThreads, 0, st>>>(strip_mat(M), sp, sc, sv, at, perm,
                                                             icol, M.col, M.val);
      PDLP_LAUNCH_CHECK();
    };
    fill(P->AT, tptr, sort.rowk, val, pos, P->perm_n, P->perm_m ? inv_m : nullptr);
    fill(P->A, ptr, col, val, nullptr, P->perm_m, P->perm_n ? inv_n : nullptr);
    if (most > 0) {
      k_gather<<<dim3(grid_for((long)most), lists), kThreads, 0, st>>>(list);
      PDLP_LAUNCH_CHECK();
    }
    P->fp32 = std::make_shared<Fp32Order>();
    if (for_fp32) {
      fp32_order_upload(*P, fp32_host.get(), *P->fp32, st);
    } else {
      P->fp32->ptr.assign(prob->constraint_matrix_row_pointers,
                          prob->constraint_matrix_row_pointers + m + 1);
      P->fp32->tptr = std::move(tp);
    }
  } else {
    auto h2d = [&](void *dst, const void *src, size_t b) {
      if (b) PDLP_CUDA(cudaMemcpyAsync(dst, src, b, cudaMemcpyHostToDevice, st));
    };
    h2d(P->A.ptr, prob->constraint_matrix_row_pointers, (vm + 1) * 4);
    h2d(P->A.col, prob->constraint_matrix_col_indices, (size_t)nnz * 4);
    h2d(P->A.val, prob->constraint_matrix_values, (size_t)nnz * 8);
    device_transpose(m, n, nnz, P->A.ptr, P->A.col, P->A.val, P->AT.ptr, P->AT.col, P->AT.val,
                     scratch.p, st);
    for (const Vec &v : vecs) h2d(v.dst, v.src, v.count * 8);
  }
  PDLP_CUDA(cudaStreamSynchronize(st));  // host staging (plans) must outlive the copies
  return P.release();
}


template class Solve<double, double>;

}  // namespace pdlp
