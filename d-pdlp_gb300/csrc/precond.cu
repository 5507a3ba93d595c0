// precond.cu -- diagonal rescaling of the LP on the GPU.
//
// Restates the reference's host preconditioner (src/preconditioner.c:89-273)
// as device sweeps over A (CSR) and A^T (CSR of the transpose):
//   Ruiz L-inf, l_inf_ruiz_iterations times: row maxima over A, column maxima
//     over A^T rows, r = sqrt(max) (1 where max < 1e-12), then
//     a_ij /= r_i * s_j, c /= s, bounds of x *= s, bounds of Ax /= r;
//   Pock-Chambolle: row sums of |a|^alpha over A, column sums of
//     |a|^(2-alpha) over A^T rows, sqrt, same scaling;
//   bound / objective rescaling: cb = 1/(|b| + 1), ob = 1/(|c| + 1).
// Maxima are order-free and every PC sum runs sequentially in the reference's
// accumulation order (row order of the CSR for rows, increasing row index for
// columns, which is the row order of A^T), so the scaled matrix, c, bounds
// and cumulative scalings are bit-identical to the host algorithm; only the
// two bound/objective norms are tree sums.
#include <math.h>

#include <algorithm>

#include "solver.cuh"

namespace pdlp {

constexpr double kScalingEps = 1e-12;

// one warp per row: out[r] = transform(max_k |val_k|)
__global__ void k_row_absmax(int rows, const int *__restrict__ ptr,
                             const double *__restrict__ val, double *__restrict__ out) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r = warp; r < rows; r += nwarps) {
    double mx = 0.0;
    for (int k = ptr[r] + lane; k < ptr[r + 1]; k += 32) mx = fmax(mx, fabs(val[k]));
    mx = warp_max(mx);
    if (lane == 0) out[r] = mx < kScalingEps ? 1.0 : sqrt(mx);
  }
}

__device__ __forceinline__ double pow_exact(double v, double e) {
  if (e == 1.0) return v;
  if (e == 2.0) return v * v;
  if (e == 0.0) return 1.0;
  return pow(v, e);
}

// one thread per row, sequential sum in row order
__global__ void k_row_powsum(int rows, const int *__restrict__ ptr,
                             const double *__restrict__ val, double e,
                             double *__restrict__ out) {
  long stride = (long)gridDim.x * blockDim.x;
  for (long r = blockIdx.x * (long)blockDim.x + threadIdx.x; r < rows; r += stride) {
    double s = 0.0;
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) s += pow_exact(fabs(val[k]), e);
    out[r] = s < kScalingEps ? 1.0 : sqrt(s);
  }
}

// a_k /= rs[row] * cs[col]   (products commute exactly, so A and A^T agree)
__global__ void k_scale_rows(int rows, const int *__restrict__ ptr,
                             const int *__restrict__ col, double *__restrict__ val,
                             const double *__restrict__ rs, const double *__restrict__ cs) {
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r = warp; r < rows; r += nwarps) {
    double a = rs[r];
    for (int k = ptr[r] + lane; k < ptr[r + 1]; k += 32) val[k] /= (a * cs[col[k]]);
  }
}

// ---- the same sweeps on the strip format (strip.cuh)
//
// One pass does a sweep's division and, on the values just formed, the row
// maxima of the next sweep (or the last sweep's power sums): the matrix is
// read and written once per sweep.  A lane takes a strip row from its first
// element to its last, which is also the order the power sums need; rows
// longer than an item are taken by a block, the other front rows by a warp.
// What is left is the FP64 division itself: 20M of them take about 0.3 ms at
// GB300's 0.22 per clock and SM, against 0.06 ms for the pass's bytes.
enum SweepOut { kSweepNone = 0, kSweepMax = 1, kSweepPow = 2 };

// max(m, |v|) on the bit patterns of non-negative doubles (which order like
// the values): the integer pipe instead of FP64's.  NaN counts as nothing, as
// with fmax.
__device__ __forceinline__ unsigned long long abs_max(unsigned long long m, double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  return b > m && b <= 0x7ff0000000000000ull ? b : m;
}
__device__ __forceinline__ double scale_of(double v) { return v < kScalingEps ? 1.0 : sqrt(v); }

template <bool SCALE, int OUT>
__global__ void __launch_bounds__(kThreads)
    k_strip_sweep(StripMat<double> A, double *__restrict__ val,
                  const double *__restrict__ rs, const double *__restrict__ cs, double e,
                  double *__restrict__ out) {
  __shared__ unsigned long long red[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  using U64 = unsigned long long;
  auto warp_maxu = [](U64 m) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const U64 x = __shfl_xor_sync(0xffffffffu, m, o);
      m = x > m ? x : m;
    }
    return m;
  };
  // long rows: one block each (OUT == kSweepPow leaves their sums to
  // k_front_powsum)
  for (int r = blockIdx.x; r < A.p.nlong; r += gridDim.x) {
    const double a = SCALE ? rs[r] : 1.0;
    U64 mx = 0;
    for (int k = A.ptr[r] + threadIdx.x; k < A.ptr[r + 1]; k += kThreads) {
      double v = val[k];
      if (SCALE) {
        v /= a * cs[A.col[k]];
        val[k] = v;
      }
      if (OUT == kSweepMax) mx = abs_max(mx, v);
    }
    if (OUT == kSweepMax) {
      mx = warp_maxu(mx);
      if (lane == 0) red[warp] = mx;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int q = 1; q < kThreads / 32; ++q) mx = red[q] > mx ? red[q] : mx;
        out[r] = scale_of(__longlong_as_double((long long)mx));
      }
      __syncthreads();
    }
  }
  const int W = gridDim.x * (kThreads / 32);
  const int w0 = warp * gridDim.x + blockIdx.x;
  // the other front rows: a warp each
  for (int r = A.p.nlong + w0; r < A.p.nfront; r += W) {
    const double a = SCALE ? rs[r] : 1.0;
    U64 mx = 0;
    for (int k = A.ptr[r] + lane; k < A.ptr[r + 1]; k += 32) {
      double v = val[k];
      if (SCALE) {
        v /= a * cs[A.col[k]];
        val[k] = v;
      }
      if (OUT == kSweepMax) mx = abs_max(mx, v);
    }
    if (OUT == kSweepMax) {
      mx = warp_maxu(mx);
      if (lane == 0) out[r] = scale_of(__longlong_as_double((long long)mx));
    }
  }
  for (int s = w0; s < A.p.nstrip; s += W) {
    const int o0 = A.p.off[s], n = A.p.off[s + 1] - o0;
    const StripPlace place = strip_place(A.p, A.rows, s);
    const int lg = place.lg, G = 1 << lg, row = place.row + (lane >> lg);
    const size_t at = (size_t)o0 * 32 + lane;
    const bool live = row < place.end;
    const double a = SCALE && live ? rs[row] : 1.0;
    U64 mx = 0;
    double sum = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
      const int c = A.col[at + (size_t)k * 32];
      double v = 0.0;
      if (c >= 0) {
        v = val[at + (size_t)k * 32];
        if (SCALE) {
          v /= a * cs[c];
          val[at + (size_t)k * 32] = v;
        }
      }
      if (OUT == kSweepMax) mx = abs_max(mx, v);
      if (OUT == kSweepPow) {
        // in the row's order, over its lanes (padding adds nothing)
        const double t = c >= 0 ? pow_exact(fabs(v), e) : 0.0;
        if (lg == 0) sum += t;
        else
          for (int g = 0; g < G; ++g) sum += __shfl_sync(0xffffffffu, t, (lane & ~(G - 1)) + g);
      }
    }
    if (OUT == kSweepMax) {
      for (int o = 1; o < G; o <<= 1) {
        const U64 x = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = x > mx ? x : mx;
      }
    }
    if (live && (lane & (G - 1)) == 0) {
      if (OUT == kSweepMax) out[row] = scale_of(__longlong_as_double((long long)mx));
      if (OUT == kSweepPow) out[row] = scale_of(sum);
    }
  }
}

// Power sums of the front rows, in order: a warp loads 32 terms at a time and
// adds them one after the other.
__global__ void __launch_bounds__(kThreads)
    k_front_powsum(StripMat<double> A, double e, double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  for (int r = (threadIdx.x >> 5) * gridDim.x + blockIdx.x; r < A.p.nfront;
       r += gridDim.x * (kThreads / 32)) {
    const int a = A.ptr[r], n = A.ptr[r + 1] - a;
    double s = 0.0, next = lane < n ? pow_exact(fabs(A.val[a + lane]), e) : 0.0;
    for (int k = 0; k < n; k += 32) {
      const double t = next;
      const int left = n - k;
      if (k + 32 + lane < n) next = pow_exact(fabs(A.val[a + k + 32 + lane]), e);
      if (left >= 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i) s += __shfl_sync(0xffffffffu, t, i);
      } else {
        for (int i = 0; i < left; ++i) s += __shfl_sync(0xffffffffu, t, i);
      }
    }
    if (lane == 0) out[r] = scale_of(s);
  }
}

// vectors and cumulative scalings (preconditioner.c:91-99, :149-152)
__global__ void k_scale_vectors(int n, int m, double *c, double *lv, double *uv,
                                double *lc, double *uc, double *Dc, double *Dr,
                                const double *var, const double *con) {
  long stride = (long)gridDim.x * blockDim.x;
  for (long j = blockIdx.x * (long)blockDim.x + threadIdx.x; j < n; j += stride) {
    double s = var[j];
    c[j] /= s;
    uv[j] *= s;
    lv[j] *= s;
    Dc[j] *= s;
  }
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < m; i += stride) {
    double s = con[i];
    lc[i] /= s;
    uc[i] /= s;
    Dr[i] *= s;
  }
}

__global__ void k_fill(long n, double *p, double v) {
  long stride = (long)gridDim.x * blockDim.x;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += stride) p[i] = v;
}

// squared norms for the bound / objective rescaling (preconditioner.c:226-246)
__global__ void __launch_bounds__(kThreads)
    k_bound_obj_norms(int n, int m, const double *c, const double *lc, const double *uc,
                      double *part) {
  __shared__ double red[24];
  double a[2] = {0.0, 0.0};
  long stride = (long)gridDim.x * kThreads;
  for (long i = blockIdx.x * (long)kThreads + threadIdx.x; i < m; i += stride) {
    double lo = lc[i], up = uc[i];
    if (isfinite(lo) && lo != up) a[0] += lo * lo;
    if (isfinite(up)) a[0] += up * up;
  }
  for (long j = blockIdx.x * (long)kThreads + threadIdx.x; j < n; j += stride)
    a[1] += c[j] * c[j];
  block_reduce_fields<2, 0u>(a, red);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a[0];
    part[gridDim.x + blockIdx.x] = a[1];
  }
}

__global__ void __launch_bounds__(kThreads) k_bound_obj_fin(int g, const double *part,
                                                            double *out) {
  __shared__ double sm[32];
  double b = block_fold<false>(part, g, sm);
  double o = block_fold<false>(part + g, g, sm);
  if (threadIdx.x == 0) {
    out[0] = 1.0 / (sqrt(b) + 1.0);
    out[1] = 1.0 / (sqrt(o) + 1.0);
  }
}

__global__ void k_scale_bounds_obj(int n, int m, double *c, double *lv, double *uv,
                                   double *lc, double *uc, const double *cbob) {
  double cb = cbob[0], ob = cbob[1];
  long stride = (long)gridDim.x * blockDim.x;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < m; i += stride) {
    lc[i] *= cb;
    uc[i] *= cb;
  }
  for (long j = blockIdx.x * (long)blockDim.x + threadIdx.x; j < n; j += stride) {
    lv[j] *= cb;
    uv[j] *= cb;
    c[j] *= ob;
  }
}

static int warp_grid(int rows) {
  long w = rows;  // one warp per row
  long b = (w * 32 + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  long cap = (long)kNumSms * 16;
  return (int)(b < cap ? b : cap);
}

void gpu_rescale(const pdhg_parameters_t &p, DevCsr &A, DevCsr &AT, double *c, double *lv,
                 double *uv, double *lc, double *uc, double *Dr, double *Dc, double *cb,
                 double *ob, double *const (&tn)[2], double *const (&tm)[2], double *part,
                 cudaStream_t st,
                 double fixed_cb, double fixed_ob) {
  const int n = A.cols, m = A.rows;
  const int gv = grid_for((long)n + m);
  k_fill<<<grid_for(m), kThreads, 0, st>>>(m, Dr, 1.0);
  k_fill<<<grid_for(n), kThreads, 0, st>>>(n, Dc, 1.0);
  PDLP_LAUNCH_CHECK();
  auto apply = [&](double *con, double *var) {
    k_scale_vectors<<<gv, kThreads, 0, st>>>(n, m, c, lv, uv, lc, uc, Dc, Dr, var, con);
    if (m) k_scale_rows<<<warp_grid(m), kThreads, 0, st>>>(m, A.ptr, A.col, A.val, con, var);
    if (n) k_scale_rows<<<warp_grid(n), kThreads, 0, st>>>(n, AT.ptr, AT.col, AT.val, var, con);
    PDLP_LAUNCH_CHECK();
  };
  double *const tmp_n = tn[0], *const tmp_m = tm[0];
  const int ruiz = p.l_inf_ruiz_iterations;
  const bool pc = p.has_pock_chambolle_alpha;
  if (A.strip.on && (ruiz > 0 || pc)) {
    // both sides' sweep from (con, var) into out_m / out_n; OUT as k_strip_sweep
    auto sweep = [&](const double *con, const double *var, int out, double *out_m,
                     double *out_n) {
      auto side = [&](DevCsr &M, const double *r, const double *c, double e, double *o) {
        if (M.strip.grid == 0) return;
        const StripMat<double> S = strip_mat(M);
        const int g = std::min(std::max(M.strip.grid, M.strip.nlong), kNumSms * 8);
#define PDLP_SWEEP(SC, O) k_strip_sweep<SC, O><<<g, kThreads, 0, st>>>(S, M.val, r, c, e, o)
        if (!con) {
          if (out == kSweepMax) PDLP_SWEEP(false, kSweepMax);
          else PDLP_SWEEP(false, kSweepPow);
        } else if (out == kSweepMax) {
          PDLP_SWEEP(true, kSweepMax);
        } else if (out == kSweepPow) {
          PDLP_SWEEP(true, kSweepPow);
        } else {
          PDLP_SWEEP(true, kSweepNone);
        }
#undef PDLP_SWEEP
        if (out == kSweepPow && M.strip.nfront)
          k_front_powsum<<<std::min((M.strip.nfront + 7) / 8, kNumSms * 8), kThreads, 0, st>>>(S, e, o);
        PDLP_LAUNCH_CHECK();
      };
      const double a = p.pock_chambolle_alpha;
      side(A, con, var, a, out_m);
      side(AT, var, con, 2.0 - a, out_n);
    };
    const int sweeps = (ruiz > 0 ? ruiz : 0) + (pc ? 1 : 0);
    auto wants = [&](int i) { return i >= sweeps ? kSweepNone : i < ruiz ? kSweepMax : kSweepPow; };
    sweep(nullptr, nullptr, wants(0), tm[0], tn[0]);
    for (int i = 0; i < sweeps; ++i) {
      double *con = tm[i & 1], *var = tn[i & 1];
      k_scale_vectors<<<gv, kThreads, 0, st>>>(n, m, c, lv, uv, lc, uc, Dc, Dr, var, con);
      PDLP_LAUNCH_CHECK();
      sweep(con, var, wants(i + 1), tm[(i + 1) & 1], tn[(i + 1) & 1]);
    }
  }
  for (int it = 0; !A.strip.on && it < ruiz; ++it) {
    if (m) k_row_absmax<<<warp_grid(m), kThreads, 0, st>>>(m, A.ptr, A.val, tmp_m);
    if (n) k_row_absmax<<<warp_grid(n), kThreads, 0, st>>>(n, AT.ptr, AT.val, tmp_n);
    PDLP_LAUNCH_CHECK();
    apply(tmp_m, tmp_n);
  }
  if (!A.strip.on && pc) {
    double a = p.pock_chambolle_alpha;
    if (m) k_row_powsum<<<grid_for(m), kThreads, 0, st>>>(m, A.ptr, A.val, a, tmp_m);
    if (n) k_row_powsum<<<grid_for(n), kThreads, 0, st>>>(n, AT.ptr, AT.val, 2.0 - a, tmp_n);
    PDLP_LAUNCH_CHECK();
    apply(tmp_m, tmp_n);
  }
  if (fixed_cb > 0.0 && fixed_ob > 0.0) {
    // refinement rounds keep the first round's bound / objective scaling
    double h[2] = {fixed_cb, fixed_ob};
    double *out = part;
    PDLP_CUDA(cudaMemcpyAsync(out, h, sizeof(h), cudaMemcpyHostToDevice, st));
    k_scale_bounds_obj<<<gv, kThreads, 0, st>>>(n, m, c, lv, uv, lc, uc, out);
    PDLP_LAUNCH_CHECK();
    PDLP_CUDA(cudaStreamSynchronize(st));
    *cb = fixed_cb;
    *ob = fixed_ob;
  } else if (p.bound_objective_rescaling) {
    int g = grid_for((long)n + m);
    if (g > kMiscPart / 2 - 2) g = kMiscPart / 2 - 2;
    double *out = part + 2 * g;
    k_bound_obj_norms<<<g, kThreads, 0, st>>>(n, m, c, lc, uc, part);
    k_bound_obj_fin<<<1, kThreads, 0, st>>>(g, part, out);
    k_scale_bounds_obj<<<gv, kThreads, 0, st>>>(n, m, c, lv, uv, lc, uc, out);
    PDLP_LAUNCH_CHECK();
    double h[2];
    PDLP_CUDA(cudaMemcpyAsync(h, out, sizeof(h), cudaMemcpyDeviceToHost, st));
    PDLP_CUDA(cudaStreamSynchronize(st));
    *cb = h[0];
    *ob = h[1];
  } else {
    *cb = 1.0;
    *ob = 1.0;
  }
}

}  // namespace pdlp
