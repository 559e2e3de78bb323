// The Method of Moving Asymptotes on the device (loadpath/mma.py:31-214, Svanberg's 2007
// formulation): the per-variable work of MMA.update and of its primal-dual interior-point
// subproblem solver, over n design variables and m <= 8 constraints, in float64.
//
//   lpb_mma_prepare   sanitised design and gradients, the moving asymptotes, move limits alfa /
//                     beta, p0 q0 P Q of the convex approximation and sum_j P_ij/ux_j + Q_ij/xl_j
//                     (loadpath/mma.py:57-103)
//   lpb_mma_sub_init  the subsolver's starting point x, xsi, eta (loadpath/mma.py:114-125)
//   lpb_mma_newton_a  one Newton step's n-sized terms: delx, diagx (kept) and the reductions
//                     gvec, GG (delx / diagx) and (GG / diagx) GG^T for the (m + 1) system
//   lpb_mma_newton_b  dx, dxsi, deta from dlam and the step-length maxima
//   lpb_mma_trial     x, xsi, eta = old + steg * d and the residual's n-sized parts at the new
//                     point (sum of squares, largest magnitude, gvec)
//   lpb_mma_finish    non-finite results back to the old design, clip to [alfa, beta]
//   lpb_mma_loop_*    the whole subproblem on the device: the loops as a graph's while node, the m-sized
//                     variables and the (m + 1) system in a state block (below)
// newton_a, newton_b and trial are the same steps for a caller whose host runs the loops, the m-sized parts of the
// residual and the (m + 1) x (m + 1) solve.
// Reductions go through fixed per-block partials summed in order (the same bits every run).
#include <math.h>

#include "lp_common.cuh"
#include "lp_mma_var.cuh"

#define LP_MMA_MAXM 8
#define LP_MMA_BLOCKS 592
#define LP_MMA_THREADS 256

namespace {

struct MVec {
  double v[LP_MMA_MAXM];
};

__device__ __forceinline__ double nan_to_num(double v, double nan, double big) {
  if (isnan(v)) return nan;
  if (isinf(v)) return v > 0 ? big : -big;
  return v;
}

// block reduction of K values per thread (sum or max per value) into part[k * nblocks + block]
template <int K>
__device__ __forceinline__ void block_reduce(double (&v)[K], const bool (&is_max)[K], double* __restrict__ part) {
  __shared__ double sh[LP_MMA_THREADS / 32][K > 0 ? K : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = v[k];
    for (int o = 16; o > 0; o >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, o);
      x = is_max[k] ? fmax(x, y) : x + y;
    }
    if (lane == 0) sh[w][k] = x;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    double x = sh[0][k];
    for (int ww = 1; ww < (int)(blockDim.x >> 5); ++ww) x = is_max[k] ? fmax(x, sh[ww][k]) : x + sh[ww][k];
    part[(long long)k * gridDim.x + blockIdx.x] = x;
  }
}

__global__ void k_mma_final(const double* __restrict__ part, int nblocks, int K, const int* __restrict__ maxmask,
                            double* __restrict__ out) {
  lp_after_launch();
  // one warp per value, blocks summed in a fixed order
  const int k = blockIdx.x;
  if (k >= K) return;
  const bool mx = maxmask[k] != 0;
  double x = mx ? -INFINITY : 0.0;
  for (int b = threadIdx.x; b < nblocks; b += 32) x = mx ? fmax(x, part[(long long)k * nblocks + b]) : x + part[(long long)k * nblocks + b];
  for (int o = 16; o > 0; o >>= 1) {
    const double y = __shfl_down_sync(0xffffffffu, x, o);
    x = mx ? fmax(x, y) : x + y;
  }
  if (threadIdx.x == 0) out[k] = x;
}

// ---- update: asymptotes and the convex approximation (loadpath/mma.py:57-103) ---------------
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS) k_mma_prepare(
    long long n, int m, double* __restrict__ x, const double* __restrict__ xmin, const double* __restrict__ xmax,
    double* __restrict__ low, double* __restrict__ upp, const double* __restrict__ xold1,
    const double* __restrict__ xold2, int init, double asyinit, double asyincr, double asydecr, double move,
    double* __restrict__ df0, double* __restrict__ df, double* __restrict__ alfa, double* __restrict__ beta,
    double* __restrict__ p0, double* __restrict__ q0, double* __restrict__ P, double* __restrict__ Q,
    double* __restrict__ part) {
  lp_after_launch();
  double acc[M];
  bool is_max[M];
#pragma unroll
  for (int i = 0; i < M; ++i) {
    acc[i] = 0.0;
    is_max[i] = false;
  }
  const double raa0 = 1e-5, albefa = 0.1;
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const double lo_b = xmin[j], hi_b = xmax[j];
    const double xj = fmin(fmax(isnan(x[j]) ? 0.5 : x[j], lo_b), hi_b);
    x[j] = xj;
    const double span = hi_b - lo_b;
    double l, u;
    if (init) {
      l = xj - asyinit * span;
      u = xj + asyinit * span;
    } else {
      const double x1 = xold1[j], x2 = xold2[j];
      const double zzz = (xj - x1) * (x1 - x2);
      const double factor = zzz > 0 ? asyincr : (zzz < 0 ? asydecr : 1.0);
      l = xj - factor * (x1 - low[j]);
      u = xj + factor * (upp[j] - x1);
      l = fmin(fmax(l, xj - 10 * span), xj - 0.01 * span);
      u = fmin(fmax(u, xj + 0.01 * span), xj + 10 * span);
    }
    low[j] = l;
    upp[j] = u;
    alfa[j] = fmax(fmax(l + albefa * (xj - l), xj - move * span), lo_b);
    beta[j] = fmin(fmin(u - albefa * (u - xj), xj + move * span), hi_b);
    const double xmami = fmax(span, 1e-5);
    const double ux1 = u - xj, xl1 = xj - l, ux2 = ux1 * ux1, xl2 = xl1 * xl1;
    const double g0 = nan_to_num(df0[j], 0.0, 1e6);
    df0[j] = g0;
    const double pp = fmax(g0, 0.0), qq = fmax(-g0, 0.0), pq0 = 0.001 * (pp + qq) + raa0 / xmami;
    p0[j] = (pp + pq0) * ux2;
    q0[j] = (qq + pq0) * xl2;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      if (i >= m) break;
      const long long ij = (long long)i * n + j;
      const double gi = nan_to_num(df[ij], 0.0, 1e6);
      df[ij] = gi;
      const double Pp = fmax(gi, 0.0), Qq = fmax(-gi, 0.0), PQ = 0.001 * (Pp + Qq) + raa0 / xmami;
      const double Pij = (Pp + PQ) * ux2, Qij = (Qq + PQ) * xl2;
      P[ij] = Pij;
      Q[ij] = Qij;
      acc[i] += Pij / ux1 + Qij / xl1;
    }
  }
  block_reduce<M>(acc, is_max, part);
}

// ---- subsolver -------------------------------------------------------------------------------
__global__ void k_mma_sub_init(long long n, const double* __restrict__ alfa, const double* __restrict__ beta,
                               double* __restrict__ xs, double* __restrict__ xsi, double* __restrict__ eta) {
  lp_after_launch();
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const double a = alfa[j], b = beta[j], x = 0.5 * (a + b);
    xs[j] = x;
    xsi[j] = fmax(1.0 / (x - a), 1.0);
    eta[j] = fmax(1.0 / (b - x), 1.0);
  }
}

struct MmaArrays {
  const double *low, *upp, *alfa, *beta, *p0, *q0, *P, *Q;
};

// reductions: gvec_i (M), bl_i = sum GG_ij delx_j / diagx_j (M), A_ik = sum GG_ij GG_kj / diagx_j
// for i <= k (M (M + 1) / 2, row-major upper triangle)
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS) k_mma_newton_a(long long n, int m, MmaArrays A,
                                                                 const double* __restrict__ xs,
                                                                 const double* __restrict__ xsi,
                                                                 const double* __restrict__ eta, MVec lam,
                                                                 double epsi, double* __restrict__ delx,
                                                                 double* __restrict__ diagx,
                                                                 double* __restrict__ part) {
  lp_after_launch();
  constexpr int K = 2 * M + M * (M + 1) / 2;
  double acc[K];
  bool is_max[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    acc[k] = 0.0;
    is_max[k] = false;
  }
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const double x = xs[j], ux1 = A.upp[j] - x, xl1 = x - A.low[j];
    const double ux2 = ux1 * ux1, xl2 = xl1 * xl1, ux3 = ux1 * ux2, xl3 = xl1 * xl2;
    double plam = A.p0[j], qlam = A.q0[j];
    double gg[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      gg[i] = 0.0;
      if (i < m) {
        const double Pij = A.P[(long long)i * n + j], Qij = A.Q[(long long)i * n + j];
        plam += Pij * lam.v[i];
        qlam += Qij * lam.v[i];
        acc[i] += Pij / ux1 + Qij / xl1;
        gg[i] = Pij / ux2 - Qij / xl2;
      }
    }
    const double xa = x - A.alfa[j], bx = A.beta[j] - x;
    const double dpsidx = plam / ux2 - qlam / xl2;
    const double dx_ = dpsidx - epsi / xa + epsi / bx;
    const double dg = 2.0 * (plam / ux3 + qlam / xl3) + xsi[j] / xa + eta[j] / bx;
    delx[j] = dx_;
    diagx[j] = dg;
    int k = 2 * M;
#pragma unroll
    for (int i = 0; i < M; ++i) {
      acc[M + i] += gg[i] * (dx_ / dg);
#pragma unroll
      for (int i2 = i; i2 < M; ++i2) acc[k++] += gg[i] * gg[i2] / dg;
    }
  }
  block_reduce<K>(acc, is_max, part);
}

// reductions (all maxima): -1.01 dxsi / xsi, -1.01 deta / eta, -1.01 dx / (x - alfa),
// 1.01 dx / (beta - x)
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS) k_mma_newton_b(long long n, int m, MmaArrays A,
                                                                 const double* __restrict__ xs,
                                                                 const double* __restrict__ xsi,
                                                                 const double* __restrict__ eta,
                                                                 const double* __restrict__ delx,
                                                                 const double* __restrict__ diagx, MVec dlam,
                                                                 double epsi, double* __restrict__ dx,
                                                                 double* __restrict__ dxsi, double* __restrict__ deta,
                                                                 double* __restrict__ part) {
  lp_after_launch();
  double acc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  const bool is_max[4] = {true, true, true, true};
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const double x = xs[j], ux1 = A.upp[j] - x, xl1 = x - A.low[j];
    const double ux2 = ux1 * ux1, xl2 = xl1 * xl1;
    double gtl = 0.0;   // (GG^T dlam)_j
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) gtl += (A.P[(long long)i * n + j] / ux2 - A.Q[(long long)i * n + j] / xl2) * dlam.v[i];
    const double dg = diagx[j];
    const double d = -delx[j] / dg - gtl / dg;
    const double xa = x - A.alfa[j], bx = A.beta[j] - x;
    const double s = xsi[j], e = eta[j];
    const double ds = -s + epsi / xa - s * d / xa;
    const double de = -e + epsi / bx + e * d / bx;
    dx[j] = d;
    dxsi[j] = ds;
    deta[j] = de;
    acc[0] = fmax(acc[0], -1.01 * ds / s);
    acc[1] = fmax(acc[1], -1.01 * de / e);
    acc[2] = fmax(acc[2], -1.01 * d / xa);
    acc[3] = fmax(acc[3], 1.01 * d / bx);
  }
  block_reduce<4>(acc, is_max, part);
}

// x, xsi, eta = old + steg * d; reductions at the new point: sum of squares of the n-sized
// residual parts (dpsidx - xsi + eta, xsi (x - alfa) - epsi, eta (beta - x) - epsi), their largest
// magnitude, and gvec_i (M)
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS) k_mma_trial(long long n, int m, MmaArrays A,
                                                              const double* __restrict__ xs0,
                                                              const double* __restrict__ xsi0,
                                                              const double* __restrict__ eta0,
                                                              const double* __restrict__ dx,
                                                              const double* __restrict__ dxsi,
                                                              const double* __restrict__ deta, double steg, MVec lam,
                                                              double epsi, double* __restrict__ xs,
                                                              double* __restrict__ xsi, double* __restrict__ eta,
                                                              double* __restrict__ part) {
  lp_after_launch();
  constexpr int K = 2 + M;
  double acc[K];
  bool is_max[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    acc[k] = 0.0;
    is_max[k] = k == 1;
  }
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    double x = xs0[j], s = xsi0[j], e = eta0[j];
    if (dx) {
      x += steg * dx[j];
      s += steg * dxsi[j];
      e += steg * deta[j];
      xs[j] = x;
      xsi[j] = s;
      eta[j] = e;
    }
    const double ux1 = A.upp[j] - x, xl1 = x - A.low[j];
    double plam = A.p0[j], qlam = A.q0[j];
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) {
        const double Pij = A.P[(long long)i * n + j], Qij = A.Q[(long long)i * n + j];
        plam += Pij * lam.v[i];
        qlam += Qij * lam.v[i];
        acc[2 + i] += Pij / ux1 + Qij / xl1;
      }
    const double r1 = plam / (ux1 * ux1) - qlam / (xl1 * xl1) - s + e;
    const double r5 = s * (x - A.alfa[j]) - epsi;
    const double r6 = e * (A.beta[j] - x) - epsi;
    acc[0] += r1 * r1 + r5 * r5 + r6 * r6;
    acc[1] = fmax(acc[1], fmax(fabs(r1), fmax(fabs(r5), fabs(r6))));
  }
  block_reduce<K>(acc, is_max, part);
}

// ---- the subproblem's loops on the device ------------------------------------------------------
// A Newton step is two passes over the variables: k_mma_maxima forms the directions and their step-length
// maxima, k_mma_move forms them again, moves the point by steg and leaves at the new point the residual's
// sums and the sums of the next Newton system. Nothing n-sized is stored between them: the directions are
// recomputed from the point and dlam, so a step reads 11 arrays and then reads 11 and writes 3, where
// newton_a, newton_b and trial move 44. Between the passes one block each (k_mma_steg, k_mma_test) does
// what the host did: step length, line search, epsi's descent, the (m + 1) system. The passes are bound by
// memory (14 MB an array at 192 x 96 x 96 variables) and the float64 units together; quotients that share a
// divisor share its inverse, corrected (lp_mma_var.cuh). An update there takes 2.97 ms; 2.76 with the products
// left uncorrected, which are off by up to twice as much as divisions; 9.98 with the host between the passes
// (half of it waiting for results).
constexpr int MMA_LOOP_BLOCKS = 296;   // two per SM

struct MmaState {
  double lam[LP_MMA_MAXM];
  double status, which, passes;        // status: 0 running, 1 done, 2 singular system
  double y[LP_MMA_MAXM], mu[LP_MMA_MAXM], s[LP_MMA_MAXM], z, zet;
  double ty[LP_MMA_MAXM], tlam[LP_MMA_MAXM], tmu[LP_MMA_MAXM], ts[LP_MMA_MAXM], tz, tzet;   // the trial point's
  double dy[LP_MMA_MAXM], dlam[LP_MMA_MAXM], dmu[LP_MMA_MAXM], ds[LP_MMA_MAXM], dz, dzet;
  double a[LP_MMA_MAXM], b[LP_MMA_MAXM], c[LP_MMA_MAXM], d[LP_MMA_MAXM], a0;
  double epsi, epsimin, norm, steg;
  int it, halvings, fresh, move;       // fresh: a new direction (its maxima are wanted); move: a trial step
};

struct MmaInit {
  double a[LP_MMA_MAXM], c[LP_MMA_MAXM], d[LP_MMA_MAXM], f[LP_MMA_MAXM], a0, epsimin;
};

struct MmaSets {
  double* v[2][3];   // x, xsi, eta of the two points
};

__global__ void k_mma_begin(MmaState* __restrict__ st, const double* __restrict__ bsum, MmaInit in, int m) {
  lp_after_launch();
  const int i = threadIdx.x;
  if (i < LP_MMA_MAXM) {
    const bool on = i < m;
    st->y[i] = st->lam[i] = st->s[i] = on ? 1.0 : 0.0;
    st->mu[i] = on ? (0.5 * in.c[i] > 1.0 || isnan(in.c[i]) ? 0.5 * in.c[i] : 1.0) : 0.0;
    st->a[i] = in.a[i];
    st->c[i] = in.c[i];
    st->d[i] = in.d[i];
    st->b[i] = on ? bsum[i] - in.f[i] : 0.0;
  }
  if (i == 0) {
    st->z = st->zet = 1.0;
    st->a0 = in.a0;
    st->epsi = 1.0;
    st->epsimin = in.epsimin;
    st->status = st->which = st->passes = 0.0;
    st->it = st->halvings = st->fresh = st->move = 0;
  }
}

__device__ __forceinline__ MmaVar mma_var(const MmaArrays& A, const MmaSets& sets, int which, long long j) {
  MmaVar v;
  v.x = (which ? sets.v[1][0] : sets.v[0][0])[j];
  v.s = (which ? sets.v[1][1] : sets.v[0][1])[j];
  v.e = (which ? sets.v[1][2] : sets.v[0][2])[j];
  v.up = A.upp[j];
  v.lo = A.low[j];
  v.al = A.alfa[j];
  v.be = A.beta[j];
  return v;
}

// maxima of -1.01 dxsi / xsi, -1.01 deta / eta, -1.01 dx / (x - alfa), 1.01 dx / (beta - x)
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS, M > 2 ? 1 : 2) k_mma_maxima(long long n, int m, MmaArrays A, MmaSets sets,
                                                                  const MmaState* __restrict__ st,
                                                                  double* __restrict__ part) {
  lp_after_launch();
  if (!st->fresh) return;
  __shared__ double lam[M], dlam[M];
  if (threadIdx.x < M) {
    lam[threadIdx.x] = st->lam[threadIdx.x];
    dlam[threadIdx.x] = st->dlam[threadIdx.x];
  }
  __syncthreads();
  const double epsi = st->epsi;
  const int which = (int)st->which;
  double acc[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  const bool is_max[4] = {true, true, true, true};
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    MmaVar v = mma_var(A, sets, which, j);
    double plam = A.p0[j], qlam = A.q0[j], gp = 0.0, gq = 0.0;
#pragma unroll
    for (int i = 0; i < M; ++i)
      if (i < m) {
        const double P = A.P[(long long)i * n + j], Q = A.Q[(long long)i * n + j];
        plam += P * lam[i];
        qlam += Q * lam[i];
        gp += P * dlam[i];
        gq += Q * dlam[i];
      }
    v.distances();
    double dx, ds, de;
    v.direction(plam, qlam, gp, gq, epsi, dx, ds, de);
    acc[0] = fmax(acc[0], -1.01 * ds / v.s);
    acc[1] = fmax(acc[1], -1.01 * de / v.e);
    acc[2] = fmax(acc[2], v.over_xa(-1.01 * dx));
    acc[3] = fmax(acc[3], v.over_bx(1.01 * dx));
  }
  block_reduce<4>(acc, is_max, part);
}

// warp sum or maximum of a value's partials (every lane gets it)
__device__ __forceinline__ double mma_part(const double* __restrict__ part, int k, bool mx) {
  double x = mx ? -INFINITY : 0.0;
  for (int b = threadIdx.x & 31; b < MMA_LOOP_BLOCKS; b += 32) {
    const double y = part[k * MMA_LOOP_BLOCKS + b];
    x = mx ? fmax(x, y) : x + y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double y = __shfl_xor_sync(0xffffffffu, x, o);
    x = mx ? fmax(x, y) : x + y;
  }
  return x;
}

// the step length of a fresh direction (the largest keeping the variables positive and inside their
// limits, at most 1), and the trial point's m-sized variables
__global__ void __launch_bounds__(128) k_mma_steg(MmaState* __restrict__ st, const double* __restrict__ part, int m) {
  lp_after_launch();
  if (!st->move) return;
  __shared__ double mx[4];
  const int w = threadIdx.x >> 5;
  if (st->fresh) {
    const double v = mma_part(part, w, true);
    if ((threadIdx.x & 31) == 0) mx[w] = v;
  }
  __syncthreads();
  if (threadIdx.x) return;
  if (st->fresh) {
    // (comparisons in this order: a NaN among the m-sized ratios never shortens the step)
    double t = -INFINITY;
    bool nan = false;
    auto ratio = [&](double d, double v) {
      const double r = -1.01 * d / v;
      nan = nan || isnan(r);
      if (r > t) t = r;
    };
    for (int i = 0; i < m; ++i) {
      ratio(st->dy[i], st->y[i]);
      ratio(st->dlam[i], st->lam[i]);
      ratio(st->dmu[i], st->mu[i]);
      ratio(st->ds[i], st->s[i]);
    }
    ratio(st->dz, st->z);
    ratio(st->dzet, st->zet);
    double top = mx[2];
    if (mx[3] > top) top = mx[3];
    if (!nan) {
      if (mx[0] > t) t = mx[0];
      if (mx[1] > t) t = mx[1];
      if (t > top) top = t;
    }
    if (1.0 > top) top = 1.0;
    st->steg = 1.0 / top;
  }
  const double g = st->steg;
  for (int i = 0; i < m; ++i) {
    st->ty[i] = st->y[i] + g * st->dy[i];
    st->tlam[i] = st->lam[i] + g * st->dlam[i];
    st->tmu[i] = st->mu[i] + g * st->dmu[i];
    st->ts[i] = st->s[i] + g * st->ds[i];
  }
  st->tz = st->z + g * st->dz;
  st->tzet = st->zet + g * st->dzet;
}

// the point moved by steg along its direction (move) into the other set, or as it is; sums there: the residual's
// squares, its largest magnitude, gvec (M), GG (delx / diagx) (M), (GG / diagx) GG^T (upper triangle)
template <int M>
__global__ void __launch_bounds__(LP_MMA_THREADS, M > 2 ? 1 : 2) k_mma_move(long long n, int m, MmaArrays A, MmaSets sets,
                                                                const MmaState* __restrict__ st,
                                                                double* __restrict__ part) {
  lp_after_launch();
  constexpr int K = 2 + 2 * M + M * (M + 1) / 2;
  const bool move = st->move;
  __shared__ double lam[M], dlam[M], tlam[M];
  if (threadIdx.x < M) {
    lam[threadIdx.x] = st->lam[threadIdx.x];
    dlam[threadIdx.x] = st->dlam[threadIdx.x];
    tlam[threadIdx.x] = move ? st->tlam[threadIdx.x] : st->lam[threadIdx.x];
  }
  __syncthreads();
  const double epsi = st->epsi, steg = st->steg;
  const int which = (int)st->which;
  double acc[K];
  bool is_max[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    acc[k] = 0.0;
    is_max[k] = k == 1;
  }
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    MmaVar v = mma_var(A, sets, which, j);
    const double p0 = A.p0[j], q0 = A.q0[j];
    double plam = p0, qlam = q0, gp = 0.0, gq = 0.0, pnew = p0, qnew = q0, P[M], Q[M];
#pragma unroll
    for (int i = 0; i < M; ++i) {
      P[i] = Q[i] = 0.0;
      if (i < m) {
        P[i] = A.P[(long long)i * n + j];
        Q[i] = A.Q[(long long)i * n + j];
        plam += P[i] * lam[i];
        qlam += Q[i] * lam[i];
        gp += P[i] * dlam[i];
        gq += Q[i] * dlam[i];
        pnew += P[i] * tlam[i];
        qnew += Q[i] * tlam[i];
      }
    }
    if (move) {
      v.distances();
      double dx, ds, de;
      v.direction(plam, qlam, gp, gq, epsi, dx, ds, de);
      v.x += steg * dx;
      v.s += steg * ds;
      v.e += steg * de;
      (which ? sets.v[0][0] : sets.v[1][0])[j] = v.x;
      (which ? sets.v[0][1] : sets.v[1][1])[j] = v.s;
      (which ? sets.v[0][2] : sets.v[1][2])[j] = v.e;
    }
    v.distances();
    const double r1 = v.over_ux2(pnew) - v.over_xl2(qnew) - v.s + v.e;
    const double r5 = v.s * v.xa - epsi, r6 = v.e * v.bx - epsi;
    acc[0] += r1 * r1 + r5 * r5 + r6 * r6;
    acc[1] = fmax(acc[1], fmax(fabs(r1), fmax(fabs(r5), fabs(r6))));
    double delx, diagx;
    v.newton(pnew, qnew, epsi, delx, diagx);
    const double idg = 1.0 / diagx, t = lp_quotient(delx, diagx, idg);
    int k = 2 + 2 * M;
    double gg[M];
#pragma unroll
    for (int i = 0; i < M; ++i) gg[i] = v.over_ux2(P[i]) - v.over_xl2(Q[i]);
#pragma unroll
    for (int i = 0; i < M; ++i) {
      acc[2 + i] += v.over_ux(P[i]) + v.over_xl(Q[i]);
      acc[2 + M + i] += gg[i] * t;
#pragma unroll
      for (int i2 = i; i2 < M; ++i2) acc[k++] += lp_quotient(gg[i] * gg[i2], diagx, idg);
    }
  }
  block_reduce<K>(acc, is_max, part);
}

// (m + 1) x (m + 1) system by elimination with partial pivoting; false when a pivot is exactly zero
__device__ bool mma_solve(double (*a)[LP_MMA_MAXM + 2], int n) {
  for (int k = 0; k < n; ++k) {
    int p = k;
    for (int r = k + 1; r < n; ++r)
      if (fabs(a[r][k]) > fabs(a[p][k])) p = r;
    if (a[p][k] == 0.0) return false;
    if (p != k)
      for (int c = k; c <= n; ++c) {
        const double t = a[k][c];
        a[k][c] = a[p][c];
        a[p][c] = t;
      }
    for (int r = k + 1; r < n; ++r) {
      const double f = a[r][k] / a[k][k];
      for (int c = k + 1; c <= n; ++c) a[r][c] -= f * a[k][c];
    }
  }
  for (int k = n - 1; k >= 0; --k) {
    double t = a[k][n];
    for (int c = k + 1; c < n; ++c) t -= a[k][c] * a[c][n];
    a[k][n] = t / a[k][k];
  }
  return true;
}

// After k_mma_move: accept the trial point or halve its step; then the next Newton system, or the next epsi
// (loadpath/mma.py:126-214, the loops flattened: one pass of them per body of the while node)
__global__ void __launch_bounds__(256) k_mma_test(cudaGraphConditionalHandle handle, MmaState* __restrict__ st,
                                                  const double* __restrict__ part, int m, int M) {
  lp_after_launch();
  __shared__ double o[2 + 2 * LP_MMA_MAXM + LP_MMA_MAXM * (LP_MMA_MAXM + 1) / 2];
  __shared__ double sys[LP_MMA_MAXM + 1][LP_MMA_MAXM + 2];
  const int K = 2 + 2 * M + M * (M + 1) / 2;
  for (int k = threadIdx.x >> 5; k < K; k += 8) {
    const double v = mma_part(part, k, k == 1);
    if ((threadIdx.x & 31) == 0) o[k] = v;
  }
  __syncthreads();
  if (threadIdx.x) return;
  const bool move = st->move;
  const double *y = move ? st->ty : st->y, *lam = move ? st->tlam : st->lam, *mu = move ? st->tmu : st->mu;
  const double *s = move ? st->ts : st->s, z = move ? st->tz : st->z, zet = move ? st->tzet : st->zet;
  const double epsi = st->epsi, *gvec = o + 2, *bl = o + 2 + M;
  st->passes += 1.0;
  // norm and largest magnitude of the residual
  double ss = 0.0, top = 0.0, al = 0.0;
  bool nan = false;
  auto part_of = [&](double r) {
    ss += r * r;
    nan = nan || isnan(r);
    if (fabs(r) > top) top = fabs(r);
  };
  for (int i = 0; i < m; ++i) {
    part_of(st->c[i] + st->d[i] * y[i] - mu[i] - lam[i]);
    al += st->a[i] * lam[i];
    part_of(gvec[i] - st->a[i] * z - y[i] + s[i] - st->b[i]);
    part_of(mu[i] * y[i] - epsi);
    part_of(lam[i] * s[i] - epsi);
  }
  part_of(st->a0 - zet - al);
  part_of(zet * z - epsi);
  const double norm = sqrt(o[0] + ss), rmax = !nan && top > o[1] ? top : o[1];
  bool go = true;
  if (move) {
    if (!(norm < 2.0 * st->norm) && ++st->halvings < 50) {
      st->steg *= 0.5;
      st->fresh = 0;
      cudaGraphSetConditional(handle, 1u);
      return;
    }
    for (int i = 0; i < m; ++i) {
      st->y[i] = y[i];
      st->lam[i] = lam[i];
      st->mu[i] = mu[i];
      st->s[i] = s[i];
    }
    st->z = z;
    st->zet = zet;
    st->which = 1.0 - st->which;
  } else {
    st->it = 0;
  }
  st->norm = norm;
  y = st->y;
  lam = st->lam;
  mu = st->mu;
  s = st->s;
  if (rmax > 0.9 * epsi && st->it < 200) {
    st->it += 1;
    const int n = m + 1;
    int k = 2 + 2 * M;
    for (int i = 0; i < M; ++i)
      for (int j = i; j < M; ++j, ++k)
        if (j < m) sys[i][j] = sys[j][i] = o[k];
    for (int i = 0; i < m; ++i) {
      const double dely = st->c[i] + st->d[i] * y[i] - lam[i] - epsi / y[i], diagy = st->d[i] + mu[i] / y[i];
      const double dellam = gvec[i] - st->a[i] * z - y[i] - st->b[i] + epsi / lam[i];
      sys[i][i] += s[i] / lam[i] + 1.0 / diagy;
      sys[i][n] = dellam + dely / diagy - bl[i];
      sys[i][m] = sys[m][i] = st->a[i];
    }
    sys[m][m] = -zet / z;
    sys[m][n] = st->a0 - al - epsi / z;
    if (mma_solve(sys, n)) {
      const double dz = sys[m][n];
      for (int i = 0; i < m; ++i) {
        const double dl = sys[i][n];
        const double dely = st->c[i] + st->d[i] * y[i] - lam[i] - epsi / y[i], diagy = st->d[i] + mu[i] / y[i];
        const double dy = -dely / diagy + dl / diagy;
        st->dlam[i] = dl;
        st->dy[i] = dy;
        st->dmu[i] = -mu[i] + epsi / y[i] - mu[i] * dy / y[i];
        st->ds[i] = -s[i] + epsi / lam[i] - s[i] * dl / lam[i];
      }
      st->dz = dz;
      st->dzet = -zet + epsi / z - zet * dz / z;
      st->fresh = st->move = 1;
      st->halvings = 0;
    } else {
      st->status = 2.0;
      go = false;
    }
  } else {
    st->epsi = epsi * 0.1;
    st->fresh = st->move = 0;
    if (!(st->epsi > st->epsimin)) {
      st->status = 1.0;
      go = false;
    }
  }
  cudaGraphSetConditional(handle, go ? 1u : 0u);
}

__global__ void k_mma_finish(long long n, const double* __restrict__ xs, const double* __restrict__ x,
                             const double* __restrict__ alfa, const double* __restrict__ beta,
                             double* __restrict__ xnew) {
  lp_after_launch();
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    double v = xs[j];
    if (!isfinite(v)) v = x[j];
    xnew[j] = fmin(fmax(v, alfa[j]), beta[j]);
  }
}

// which of a kernel's K reduced values are maxima: a small device table per layout
__device__ int g_mask_sum[64];                              // all zero: sums
__device__ int g_mask_max4[4] = {1, 1, 1, 1};
__device__ int g_mask_trial[2 + LP_MMA_MAXM] = {0, 1};   // [1]: the largest magnitude

static int final_reduce(const double* part, int K, const int* mask_dev, double* out, cudaStream_t st) {
  lp_launch(k_mma_final, K, 32, 0, st, part, LP_MMA_BLOCKS, K, mask_dev, out);
  return LP_OK;
}

template <typename T>
static const int* dev_addr(T& sym) {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, sym) != cudaSuccess) return nullptr;
  return static_cast<const int*>(p);
}

static int mma_m_template(int m) {
  if (m <= 1) return 1;
  if (m <= 2) return 2;
  if (m <= 4) return 4;
  return 8;
}

static MVec mvec(const double* h, int m) {
  MVec v;
  for (int i = 0; i < LP_MMA_MAXM; ++i) v.v[i] = (h && i < m) ? h[i] : 0.0;
  return v;
}

}  // namespace

#define LP_ST ((cudaStream_t)stream)
#define MMA_GRID LP_MMA_BLOCKS, LP_MMA_THREADS, 0, LP_ST
#define MMA_DISPATCH(KERNEL, ...)                                              \
  switch (mma_m_template(m)) {                                                  \
    case 1: lp_launch(KERNEL<1>, MMA_GRID, __VA_ARGS__); break;                        \
    case 2: lp_launch(KERNEL<2>, MMA_GRID, __VA_ARGS__); break;                        \
    case 4: lp_launch(KERNEL<4>, MMA_GRID, __VA_ARGS__); break;                        \
    default: lp_launch(KERNEL<8>, MMA_GRID, __VA_ARGS__); break;                       \
  }

extern "C" {

// part: scratch of at least lpb_mma_part_len(m) doubles: LP_MMA_BLOCKS partials for each value
// of the widest reduction any pass makes (prepare M, newton_a 2M + M(M+1)/2, newton_b 4,
// trial 2 + M, M = m rounded up to 1, 2, 4 or 8)
long long lpb_mma_part_len(int m) {
  const int M = mma_m_template(m);
  int K = 2 * M + M * (M + 1) / 2;
  if (K < 4) K = 4;
  if (K < 2 + M) K = 2 + M;
  return (long long)K * LP_MMA_BLOCKS;
}

int lpb_mma_prepare(long long n, int m, double* x, const double* xmin, const double* xmax, double* low, double* upp,
                    const double* xold1, const double* xold2, int init, double asyinit, double asyincr,
                    double asydecr, double move, double* df0, double* df, double* alfa, double* beta, double* p0,
                    double* q0, double* P, double* Q, double* part, double* bsum, void* stream) {
  if (n < 1 || m < 1 || m > LP_MMA_MAXM || !x || !xmin || !xmax || !low || !upp || !df0 || !df || !alfa || !beta ||
      !p0 || !q0 || !P || !Q || !part || !bsum)
    return LP_ERR_ARG;
  if (!init && (!xold1 || !xold2)) return LP_ERR_ARG;
  const int* mask = dev_addr(g_mask_sum);
  if (!mask) return LP_ERR_LAUNCH;
  MMA_DISPATCH(k_mma_prepare, n, m, x, xmin, xmax, low, upp, xold1, xold2, init, asyinit, asyincr, asydecr, move,
               df0, df, alfa, beta, p0, q0, P, Q, part)
  final_reduce(part, mma_m_template(m), mask, bsum, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_mma_sub_init(long long n, const double* alfa, const double* beta, double* xs, double* xsi, double* eta,
                     void* stream) {
  if (n < 1 || !alfa || !beta || !xs || !xsi || !eta) return LP_ERR_ARG;
  lp_launch(k_mma_sub_init, MMA_GRID, n, alfa, beta, xs, xsi, eta);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// out: gvec (M values), GG (delx / diagx) (M), (GG / diagx) GG^T upper triangle (M (M + 1) / 2),
// M = m rounded up to 1, 2, 4 or 8; lam: HOST pointer to m doubles
int lpb_mma_newton_a(long long n, int m, const double* low, const double* upp, const double* alfa,
                     const double* beta, const double* p0, const double* q0, const double* P, const double* Q,
                     const double* xs, const double* xsi, const double* eta, const double* lam, double epsi,
                     double* delx, double* diagx, double* part, double* out, void* stream) {
  if (n < 1 || m < 1 || m > LP_MMA_MAXM || !low || !upp || !alfa || !beta || !p0 || !q0 || !P || !Q || !xs || !xsi ||
      !eta || !lam || !delx || !diagx || !part || !out)
    return LP_ERR_ARG;
  const int* mask = dev_addr(g_mask_sum);
  if (!mask) return LP_ERR_LAUNCH;
  const MmaArrays A = {low, upp, alfa, beta, p0, q0, P, Q};
  const MVec lv = mvec(lam, m);
  MMA_DISPATCH(k_mma_newton_a, n, m, A, xs, xsi, eta, lv, epsi, delx, diagx, part)
  const int M = mma_m_template(m);
  final_reduce(part, 2 * M + M * (M + 1) / 2, mask, out, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// out: the four step-length maxima; dlam: HOST pointer to m doubles
int lpb_mma_newton_b(long long n, int m, const double* low, const double* upp, const double* alfa,
                     const double* beta, const double* P, const double* Q, const double* xs, const double* xsi,
                     const double* eta, const double* delx, const double* diagx, const double* dlam, double epsi,
                     double* dx, double* dxsi, double* deta, double* part, double* out, void* stream) {
  if (n < 1 || m < 1 || m > LP_MMA_MAXM || !low || !upp || !alfa || !beta || !P || !Q || !xs || !xsi || !eta ||
      !delx || !diagx || !dlam || !dx || !dxsi || !deta || !part || !out)
    return LP_ERR_ARG;
  const int* mask = dev_addr(g_mask_max4);
  if (!mask) return LP_ERR_LAUNCH;
  const MmaArrays A = {low, upp, alfa, beta, nullptr, nullptr, P, Q};
  const MVec dl = mvec(dlam, m);
  MMA_DISPATCH(k_mma_newton_b, n, m, A, xs, xsi, eta, delx, diagx, dl, epsi, dx, dxsi, deta, part)
  final_reduce(part, 4, mask, out, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// x, xsi, eta = (x0, xsi0, eta0) + steg (dx, dxsi, deta) (dx NULL: the residual at x0, nothing
// written); out: sum of squares, largest magnitude, gvec (M); lam: HOST pointer to m doubles
int lpb_mma_trial(long long n, int m, const double* low, const double* upp, const double* alfa, const double* beta,
                  const double* p0, const double* q0, const double* P, const double* Q, const double* xs0,
                  const double* xsi0, const double* eta0, const double* dx, const double* dxsi, const double* deta,
                  double steg, const double* lam, double epsi, double* xs, double* xsi, double* eta, double* part,
                  double* out, void* stream) {
  if (n < 1 || m < 1 || m > LP_MMA_MAXM || !low || !upp || !alfa || !beta || !p0 || !q0 || !P || !Q || !xs0 ||
      !xsi0 || !eta0 || !lam || !part || !out)
    return LP_ERR_ARG;
  if (dx && (!dxsi || !deta || !xs || !xsi || !eta)) return LP_ERR_ARG;
  const int* mask = dev_addr(g_mask_trial);
  if (!mask) return LP_ERR_LAUNCH;
  const MmaArrays A = {low, upp, alfa, beta, p0, q0, P, Q};
  const MVec lv = mvec(lam, m);
  MMA_DISPATCH(k_mma_trial, n, m, A, xs0, xsi0, eta0, dx, dxsi, deta, steg, lv, epsi, xs, xsi, eta, part)
  final_reduce(part, 2 + mma_m_template(m), mask, out, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// ---- the subproblem as a device-side loop ----
// doubles of the state block: [0, m) lam, [8] status (1 done, 2 singular Newton system), [9] the set that
// holds the result, [10] bodies run
int lpb_mma_state_len(void) { return (int)((sizeof(MmaState) + 7) / 8); }

// the starting state: b = bsum - f, y = lam = s = z = zet = 1, mu = max(1, c / 2); a, c, d, f: HOST pointers to m
int lpb_mma_loop_begin(int m, double* state, const double* bsum, const double* a, const double* c, const double* d,
                       const double* f, double a0, double epsimin, void* stream) {
  if (m < 1 || m > LP_MMA_MAXM || !state || !bsum || !a || !c || !d || !f) return LP_ERR_ARG;
  MmaInit in{};
  for (int i = 0; i < m; ++i) {
    in.a[i] = a[i];
    in.c[i] = c[i];
    in.d[i] = d[i];
    in.f[i] = f[i];
  }
  in.a0 = a0;
  in.epsimin = epsimin;
  lp_launch(k_mma_begin, 1, 32, 0, LP_ST, reinterpret_cast<MmaState*>(state), bsum, in, m);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// one body of the loop (four launches), recorded between lpb_while_begin, which gave handle, and
// lpb_while_end; the first set holds the starting point, part: lpb_mma_part_len(m) doubles
int lpb_mma_loop_body(long long handle, long long n, int m, const double* low, const double* upp, const double* alfa,
                      const double* beta, const double* p0, const double* q0, const double* P, const double* Q,
                      double* x0, double* xsi0, double* eta0, double* x1, double* xsi1, double* eta1, double* state,
                      double* part, void* stream) {
  if (n < 1 || m < 1 || m > LP_MMA_MAXM || !low || !upp || !alfa || !beta || !p0 || !q0 || !P || !Q || !x0 || !xsi0 ||
      !eta0 || !x1 || !xsi1 || !eta1 || !state || !part)
    return LP_ERR_ARG;
  const MmaArrays A = {low, upp, alfa, beta, p0, q0, P, Q};
  const MmaSets sets = {{{x0, xsi0, eta0}, {x1, xsi1, eta1}}};
  MmaState* st = reinterpret_cast<MmaState*>(state);
  const int M = mma_m_template(m);
#define MMA_LOOP(KERNEL)                                                                                       \
  switch (M) {                                                                                                 \
    case 1: lp_launch(KERNEL<1>, MMA_LOOP_BLOCKS, LP_MMA_THREADS, 0, LP_ST, n, m, A, sets, st, part); break;   \
    case 2: lp_launch(KERNEL<2>, MMA_LOOP_BLOCKS, LP_MMA_THREADS, 0, LP_ST, n, m, A, sets, st, part); break;   \
    case 4: lp_launch(KERNEL<4>, MMA_LOOP_BLOCKS, LP_MMA_THREADS, 0, LP_ST, n, m, A, sets, st, part); break;   \
    default: lp_launch(KERNEL<8>, MMA_LOOP_BLOCKS, LP_MMA_THREADS, 0, LP_ST, n, m, A, sets, st, part); break;  \
  }
  MMA_LOOP(k_mma_maxima)
  lp_launch(k_mma_steg, 1, 128, 0, LP_ST, st, part, m);
  MMA_LOOP(k_mma_move)
  lp_launch(k_mma_test, 1, 256, 0, LP_ST, (cudaGraphConditionalHandle)handle, st, part, m, M);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// xnew = clip(finite(xs) ? xs : x, alfa, beta)
int lpb_mma_finish(long long n, const double* xs, const double* x, const double* alfa, const double* beta,
                   double* xnew, void* stream) {
  if (n < 1 || !xs || !x || !alfa || !beta || !xnew) return LP_ERR_ARG;
  lp_launch(k_mma_finish, MMA_GRID, n, xs, x, alfa, beta, xnew);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

}  // extern "C"
