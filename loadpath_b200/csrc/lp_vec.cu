// Vector passes of the V-cycle and the PCG (loadpath/mgops.py:302-360, :557-585, :593-773):
// Chebyshev updates, fused CG step with |r|^2, p = z + beta p, dots, casts, and the grid
// transfers (residual -> pad -> full-weighting restriction -> coarse mask; prolongation ->
// fine mask -> add).
//
// Reductions are deterministic: a fixed number of blocks (LP_RED_BLOCKS) each write a
// partial sum and one block adds the partials in order, so a given input always gives the
// same bits. Scalars the solver needs between kernels (rz, pap, |r|^2, alpha, beta) live in
// device memory so an iteration never waits on the host.
#include "lp_common.cuh"

#define LP_RED_BLOCKS 592   // 4 per SM on 148 SMs
#define LP_RED_THREADS 512

namespace {

template <typename T>
struct V4ld;
template <>
struct V4ld<float> {
  static __device__ __forceinline__ void ld(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
  static __device__ __forceinline__ void st(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct V4ld<double> {
  static __device__ __forceinline__ void ld(const double* p, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  }
  static __device__ __forceinline__ void st(double* p, const double (&v)[4]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
  }
};


template <typename Ta, typename Tb>
__global__ void k_dot_partial(const Ta* __restrict__ a, const Tb* __restrict__ b, long long n,
                              double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    s += (double)a[i] * (double)b[i];
  s = lp_block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out[0] = sum(part); optional: out_sqrt = sqrt(sum)
__global__ void k_sum_final(const double* __restrict__ part, int n, double* __restrict__ out) {
  lp_after_launch();
  __shared__ double sh[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  s = lp_block_sum(s, sh);
  if (threadIdx.x == 0) *out = s;
}

// x += alpha p ; r -= alpha ap ; r32 = (float) r ; partial |r|^2. alpha = num / den.
__global__ void k_cg_step(double* __restrict__ x, double* __restrict__ r, const double* __restrict__ p,
                          const double* __restrict__ ap, float* __restrict__ r32, long long n,
                          const double* __restrict__ num, const double* __restrict__ den, double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  const double alpha = (*num) / (*den);
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] += alpha * p[i];
    double ri = r[i] - alpha * ap[i];
    r[i] = ri;
    if (r32) r32[i] = (float)ri;
    s += ri * ri;
  }
  s = lp_block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// p = z + (num / den) p, z in float32 or float64
template <typename Tz>
__global__ void k_xpby(double* __restrict__ p, const Tz* __restrict__ z, long long n, const double* __restrict__ num,
                       const double* __restrict__ den) {
  lp_after_launch();
  const double beta = (*num) / (*den);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    p[i] = (double)z[i] + beta * p[i];
}

template <typename Ta, typename Tb>
__global__ void k_cast(Tb* __restrict__ out, const Ta* __restrict__ a, long long n) {
  lp_after_launch();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = (Tb)a[i];
}

// out = a x + b y
template <typename T>
__global__ void k_axpby(T* __restrict__ out, T a, const T* __restrict__ x, T b, const T* __restrict__ y, long long n) {
  lp_after_launch();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = a * x[i] + (y ? b * y[i] : T(0));
}

// Smoother coefficients live in device memory (written by k_cheb_coef after the power
// iteration), so a V-cycle never needs lmax on the host and a captured V-cycle stays valid when
// the hierarchy is rebuilt: coef[1] = 1 / theta, coef[2 + 2k], coef[3 + 2k] = c1, c2 of step k.

// Chebyshev start from zero: x = 0; r = b; d = (dinv b) s        (loadpath/mgops.py:321-328)
template <typename T>
__global__ void k_cheb_start(const T* __restrict__ b, const T* __restrict__ dinv, const double* __restrict__ coef,
                             T* __restrict__ x, T* __restrict__ r, T* __restrict__ d, long long n) {
  lp_after_launch();
  const T s = (T)coef[1];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    T bi = b[i];
    x[i] = T(0);
    r[i] = bi;
    d[i] = (dinv[i] * bi) * s;
  }
}

// r = b - ax; d = s dinv r                                        (loadpath/mgops.py:314-319)
template <typename T>
__global__ void k_residual_scaled(const T* __restrict__ b, const T* __restrict__ ax, const T* __restrict__ dinv,
                                  const double* __restrict__ coef, T* __restrict__ r, T* __restrict__ d, long long n) {
  lp_after_launch();
  const T s = (T)coef[1];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    T ri, di;
    lp_residual_scaled_v(b[i], ax[i], dinv[i], s, ri, di);
    r[i] = ri;
    d[i] = di;
  }
}

// x += d; unless last: r -= ad; d = c1 d + c2 dinv r             (loadpath/mgops.py:334-343)
template <typename T>
__global__ void k_cheb(T* __restrict__ x, T* __restrict__ d, T* __restrict__ r, const T* __restrict__ ad,
                       const T* __restrict__ dinv, const double* __restrict__ coef, int step, int last, long long n) {
  lp_after_launch();
  const T c1 = (T)coef[2 + 2 * step], c2 = (T)coef[3 + 2 * step];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    T di = d[i];
    x[i] += di;
    if (!last) {
      T ri = r[i] - ad[i];
      r[i] = ri;
      d[i] = c1 * di + c2 * dinv[i] * ri;
    }
  }
}

// lmax and the Chebyshev coefficients from the power iteration's dots (loadpath/mg.py:771-794,
// :796-821): lmax = safety * max(v.Av of the last step, 1e-12), or 2 when some |v|^2 was 0;
// the interval is [lmax / 30, lmax]. One thread, float64 throughout.
__global__ void k_cheb_coef(double* __restrict__ coef, const double* __restrict__ vv, const double* __restrict__ vav,
                            int its, int degree, double safety) {
  lp_after_launch();
  bool zero = false;
  for (int k = 0; k < its; ++k) zero = zero || vv[k] == 0.0;
  lp_cheb_coef(coef, vav[its - 1], zero, degree, safety);
}

// Degree-2 Chebyshev in two passes per smoothing (the reference's default degree). With
// d' = c1 d + c2 dinv (r - A d) (step 0's update) the two steps give x + d + d', formed here in
// the reference's order ((x + d) + d', and 0 + d = d exactly), so the result is the same bits as
// the step-by-step form while r and d are never rewritten.
// from zero, pass 1: d = (dinv b) s                               (loadpath/mgops.py:321-328)
template <typename T>
__global__ void k_cheb_d_start(const T* __restrict__ b, const T* __restrict__ dinv, const double* __restrict__ coef,
                               T* __restrict__ d, long long n) {
  lp_after_launch();
  const T s = (T)coef[1];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    d[i] = (dinv[i] * b[i]) * s;
}

// from zero, pass 2 (ad = A d): x = d + (c1 d + c2 dinv (b - ad))
template <typename T>
__global__ void k_cheb2_zero(T* __restrict__ x, const T* __restrict__ b, const T* __restrict__ ad,
                             const T* __restrict__ d, const T* __restrict__ dinv, const double* __restrict__ coef,
                             long long n) {
  lp_after_launch();
  const T c1 = (T)coef[2], c2 = (T)coef[3];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    x[i] = lp_cheb2_zero_v(d[i], b[i], ad[i], dinv[i], c1, c2);
}

// from x (after lpb_residual_scaled: r = b - A x, d = s dinv r; ad = A d):
// x = (x + d) + (c1 d + c2 dinv (r - ad))
template <typename T>
__global__ void k_cheb2(T* __restrict__ x, const T* __restrict__ d, const T* __restrict__ r, const T* __restrict__ ad,
                        const T* __restrict__ dinv, const double* __restrict__ coef, long long n) {
  lp_after_launch();
  const T c1 = (T)coef[2], c2 = (T)coef[3];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    x[i] = lp_cheb2_v(x[i], d[i], r[i], ad[i], dinv[i], c1, c2);
}

// damped Jacobi: x += omega dinv (b - ax), x = 0 start handled by the caller
template <typename T>
__global__ void k_jacobi(T* __restrict__ x, const T* __restrict__ b, const T* __restrict__ ax,
                         const T* __restrict__ dinv, T omega, int from_zero, long long n) {
  lp_after_launch();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (from_zero)
      x[i] = omega * dinv[i] * b[i];
    else
      x[i] += omega * dinv[i] * (b[i] - ax[i]);
  }
}

// ---- grid transfers by z chunks -----------------------------------------------------------
// One thread per (x, y) node column and chunk of four z planes (x fastest across threads), the
// chunk's values moved with 16-byte loads and stores, the trilinear weights applied separably
// (z inside a column first).

// rc = restrict(((b - ax) * m) zero-padded) * cm (loadpath/mgops.py:666-711). One warp per component of
// 15 coarse columns X0..X0+14 of one coarse row Y and chunk C (coarse planes 4C..4C+3): lane l
// reads fine column x = 2 X0 - 1 + l (rows 2Y - 1 .. 2Y + 1, fine planes 8C - 1 .. 8C + 7), so a
// warp's loads are 32 consecutive 16-byte chunk rows; the lane restricts z and y in registers,
// and the odd lanes (x = 2X) finish x with their two neighbours' sums by shuffles and store, with d
// also the first direction d = (dinv rc) s of the smoothing that starts from rc (k_cheb_d_start's
// values: a pass over the coarse field less, 3 us on the coarse levels). blockIdx.y: the column.
// Bound by the latency of its loads on all but the largest levels: the three rows' loads are in flight
// together, and the components are different warps' (float32, below 128 x 64 x 64 cells: 4.9 us, a row at a
// time for all components 6.6; below 64 x 32 x 32: 2.9 and 5.9; 256 x 128 x 128: 34.0 and 33.7).
constexpr int R4_COLS = 15;   // coarse columns per warp

template <typename T>
__global__ void __launch_bounds__(128) k_restrict4(T* __restrict__ rc, T* __restrict__ d, const T* __restrict__ dinv,
                                                   const double* __restrict__ coef, const T* __restrict__ b,
                                                   const T* __restrict__ ax, const uint8_t* __restrict__ m,
                                                   const uint8_t* __restrict__ cm, LpGrid gf, LpGrid gc) {
  lp_after_launch();
  const int CX = gc.NX(), CY = gc.NY(), CZ4 = gc.pz / 4;
  const int FX = gf.NX(), FY = gf.NY();
  const int ngx = (CX + R4_COLS - 1) / R4_COLS;
  const long long fcs = gf.comp_stride(), ccs = gc.comp_stride(), fzs = gf.node_zc_stride();
  const int lane = threadIdx.x & 31;
  const unsigned w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= 3u * ngx * CY * CZ4) return;
  const unsigned wq = w / 3, q = wq / (unsigned)ngx;
  const int i = (int)(w - 3 * wq), gx = (int)(wq - q * ngx);
  const int C = (int)(q / (unsigned)CY), Y = (int)(q - (unsigned)C * CY);
  const int X0 = gx * R4_COLS;
  const int x = 2 * X0 - 1 + lane;
  const int z0 = 8 * C;
  // a coarse level padded up past half the fine one reaches beyond the fine pitch: zeros
  const bool below = z0 >= 1 && z0 - 1 < gf.pz, lo = z0 < gf.pz, hi = z0 + 4 < gf.pz;
  long long n_lo[3], n_below[3];
  uint32_t mlo[3], mhi[3];
  uint8_t mbelow[3];
  bool in[3];
#pragma unroll
  for (int dy = 0; dy < 3; ++dy) {
    const int y = 2 * Y + dy - 1;
    in[dy] = x >= 0 && x < FX && y >= 0 && y < FY;
    n_lo[dy] = in[dy] && lo ? gf.node(x, y, z0) : 0;
    n_below[dy] = in[dy] && below ? gf.node(x, y, z0 - 1) : 0;
    mbelow[dy] = in[dy] && below ? m[n_below[dy]] : 0;
    mlo[dy] = in[dy] && lo ? *reinterpret_cast<const uint32_t*>(m + n_lo[dy]) : 0;
    mhi[dy] = in[dy] && hi ? *reinterpret_cast<const uint32_t*>(m + n_lo[dy] + fzs) : 0;
  }
  // x: coarse X = X0 + (lane - 1) / 2 on the odd lanes, from fine x - 1, x, x + 1
  const int X = X0 + ((lane - 1) >> 1);
  const bool out = (lane & 1) && lane <= 2 * R4_COLS - 1 && X < CX;
  const long long cn = out ? gc.node(X, Y, 4 * C) : 0;
  const uint32_t cmb = out ? *reinterpret_cast<const uint32_t*>(cm + cn) : 0;
  const T sd = d ? (T)coef[1] : T(0);
  const T* bi = b + (3LL * blockIdx.y + i) * fcs;
  const T* ai = ax + (3LL * blockIdx.y + i) * fcs;
  T v[3][9];
#pragma unroll
  for (int dy = 0; dy < 3; ++dy) {
    T b4[4] = {}, b5[4] = {}, a4[4] = {}, a5[4] = {}, bb = T(0), ab = T(0);
    if (in[dy] && below) {
      bb = bi[n_below[dy]];
      ab = ai[n_below[dy]];
    }
    if (in[dy] && lo) {
      V4ld<T>::ld(bi + n_lo[dy], b4);
      V4ld<T>::ld(ai + n_lo[dy], a4);
    }
    if (in[dy] && hi) {
      V4ld<T>::ld(bi + n_lo[dy] + fzs, b5);
      V4ld<T>::ld(ai + n_lo[dy] + fzs, a5);
    }
    v[dy][0] = bb - ab;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      v[dy][1 + k] = b4[k] - a4[k];
      v[dy][5 + k] = b5[k] - a5[k];
    }
  }
  T acc[4] = {};
#pragma unroll
  for (int dy = 0; dy < 3; ++dy) {
    const T wy = dy != 1 ? T(0.5) : T(1);
    if (!((mbelow[dy] >> i) & 1)) v[dy][0] = T(0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!((mlo[dy] >> (8 * k + i)) & 1)) v[dy][1 + k] = T(0);
      if (!((mhi[dy] >> (8 * k + i)) & 1)) v[dy][5 + k] = T(0);
    }
    // coarse Z = 4C + kk sums fine z = 2Z - 1, 2Z, 2Z + 1 = v[2kk], v[2kk + 1], v[2kk + 2]
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      acc[kk] += wy * (T(0.5) * v[dy][2 * kk] + v[dy][2 * kk + 1] + T(0.5) * v[dy][2 * kk + 2]);
  }
  T o[4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    const T l = __shfl_up_sync(0xffffffffu, acc[kk], 1);
    const T r = __shfl_down_sync(0xffffffffu, acc[kk], 1);
    o[kk] = ((cmb >> (8 * kk + i)) & 1) ? T(0.5) * l + acc[kk] + T(0.5) * r : T(0);
  }
  if (!out) return;
  const long long at = (3LL * blockIdx.y + i) * ccs + cn;
  V4ld<T>::st(rc + at, o);
  if (d) {
    T dv[4];
    V4ld<T>::ld(dinv + i * ccs + cn, dv);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) dv[kk] = (dv[kk] * o[kk]) * sd;
    V4ld<T>::st(d + at, dv);
  }
}

// x += prolong(xc * cm) * m for NC components of the fine nodes (x, y, 4c..4c+3): coarse planes 2c, 2c + 1,
// 2c + 2 of the one, two or four coarse columns around (x / 2, y / 2)   (loadpath/mgops.py:714-750);
// blockIdx.y: the component (NC 1), blockIdx.z: the column. Its loads too are all in flight together
// (float32, to 64 x 32 x 32 cells: 2.3 us, column by column 3.4; to 128 x 64 x 64: 7.3 and 6.6).
template <typename T, int NC>
__global__ void __launch_bounds__(128) k_prolong4(T* __restrict__ xf, const T* __restrict__ xc,
                                                  const uint8_t* __restrict__ cm, const uint8_t* __restrict__ m, LpGrid gf,
                                                  LpGrid gc) {
  lp_after_launch();
  const long long total = gf.nodes_padded() / 4, ccs = gc.comp_stride(), fcs = gf.comp_stride();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= total) return;
  int x, y, c;
  gf.node_at(4 * t, x, y, c);
  c >>= 2;
  const uint32_t mb = *reinterpret_cast<const uint32_t*>(m + 4 * t);
  const int X0 = x >> 1, Y0 = y >> 1, ox = x & 1, oy = y & 1;
  const int Z0 = 2 * c, zmax = gc.pz - 1;
  // the planes' places from the first: Z0 is even, so Z0 + 1 lies in its chunk
  const long long cz2 = gc.node(0, 0, min(Z0 + 2, zmax)) - gc.node(0, 0, Z0);
  const T w = (ox ? T(0.5) : T(1)) * (oy ? T(0.5) : T(1));
  long long cn[4];
  uint8_t cz[4][3];
  bool on[4];
#pragma unroll
  for (int ab = 0; ab < 4; ++ab) {
    on[ab] = Z0 <= zmax && (!(ab & 2) || ox) && (!(ab & 1) || oy);
    cn[ab] = on[ab] ? gc.node(X0 + (ab >> 1), Y0 + (ab & 1), Z0) : 0;
    cz[ab][0] = on[ab] ? cm[cn[ab]] : 0;
    cz[ab][1] = on[ab] ? cm[cn[ab] + 1] : 0;
    cz[ab][2] = on[ab] ? cm[cn[ab] + cz2] : 0;
  }
#pragma unroll
  for (int ii = 0; ii < NC; ++ii) {
    const int i = NC == 1 ? (int)blockIdx.y : ii;
    T* xi = xf + (3LL * blockIdx.z + i) * fcs;
    const T* ci = xc + (3LL * blockIdx.z + i) * ccs;
    T o[4], cv[4][3];
    V4ld<T>::ld(xi + 4 * t, o);
#pragma unroll
    for (int ab = 0; ab < 4; ++ab) {
      cv[ab][0] = on[ab] ? ci[cn[ab]] : T(0);
      cv[ab][1] = on[ab] ? ci[cn[ab] + 1] : T(0);
      cv[ab][2] = on[ab] ? ci[cn[ab] + cz2] : T(0);
    }
    T acc[4] = {};
#pragma unroll
    for (int ab = 0; ab < 4; ++ab) {
      T u[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) u[k] = ((cz[ab][k] >> i) & 1) ? cv[ab][k] : T(0);
      acc[0] += w * u[0];
      acc[1] += w * (T(0.5) * (u[0] + u[1]));
      acc[2] += w * u[1];
      acc[3] += w * (T(0.5) * (u[1] + u[2]));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if ((mb >> (8 * k + i)) & 1) o[k] += acc[k];
    V4ld<T>::st(xi + 4 * t, o);
  }
}

// out = u * mask (per component bit); four nodes per step (the padded node count is a multiple
// of 4), the component found by comparison, not by a 64-bit division
template <typename T>
__global__ void k_mask_field(T* __restrict__ out, const T* __restrict__ u, const uint8_t* __restrict__ m, LpGrid g,
                             int bitshift) {
  lp_after_launch();
  const long long nq = g.nodes_padded() >> 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 3 * nq; i += (long long)gridDim.x * blockDim.x) {
    const int c = i >= nq ? (i >= 2 * nq ? 2 : 1) : 0;
    const uchar4 mb = reinterpret_cast<const uchar4*>(m)[i - c * nq];
    const int sh = c + bitshift;
    T v[4];
    V4ld<T>::ld(u + 4 * i, v);
    if (!((mb.x >> sh) & 1)) v[0] = T(0);
    if (!((mb.y >> sh) & 1)) v[1] = T(0);
    if (!((mb.z >> sh) & 1)) v[2] = T(0);
    if (!((mb.w >> sh) & 1)) v[3] = T(0);
    V4ld<T>::st(out + 4 * i, v);
  }
}

// v *= 1 / sqrt(*nrm2) (power iteration normalisation); leaves v alone when the norm is 0
template <typename T>
__global__ void k_scale_rsqrt(T* __restrict__ v, long long n, const double* __restrict__ nrm2) {
  lp_after_launch();
  double s = *nrm2;
  if (s <= 0.0) return;
  T f = (T)(1.0 / sqrt(s));
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    v[i] = v[i] / (T)sqrt(s);
  (void)f;
}

// av = dinv * av * mask, four nodes per step as k_mask_field
template <typename T>
__global__ void k_dinv_mask(T* __restrict__ av, const T* __restrict__ dinv, const uint8_t* __restrict__ m, LpGrid g) {
  lp_after_launch();
  const long long nq = g.nodes_padded() >> 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 3 * nq; i += (long long)gridDim.x * blockDim.x) {
    const int c = i >= nq ? (i >= 2 * nq ? 2 : 1) : 0;
    const uchar4 mb = reinterpret_cast<const uchar4*>(m)[i - c * nq];
    T v[4], d[4];
    V4ld<T>::ld(av + 4 * i, v);
    V4ld<T>::ld(dinv + 4 * i, d);
    v[0] = ((mb.x >> c) & 1) ? d[0] * v[0] : T(0);
    v[1] = ((mb.y >> c) & 1) ? d[1] * v[1] : T(0);
    v[2] = ((mb.z >> c) & 1) ? d[2] * v[2] : T(0);
    v[3] = ((mb.w >> c) & 1) ? d[3] * v[3] : T(0);
    V4ld<T>::st(av + 4 * i, v);
  }
}


// Warm start of the PCG on the device (loadpath/mg.py:878-895), so the solve never waits on
// the host before its first iteration. sc: [0] b.b, [5] x.Ax, [6] b.x, [7] |rs|^2.
//   s = b.x / x.Ax when x.Ax > 0, else 0;  rs = b - s Ax
__device__ __forceinline__ double lp_warm_scale(const double* sc) { return sc[5] > 0.0 ? sc[6] / sc[5] : 0.0; }

__global__ void k_warm_residual(double* __restrict__ rs, const double* __restrict__ b, const double* __restrict__ ax,
                                const double* __restrict__ sc, long long n) {
  lp_after_launch();
  const double s = lp_warm_scale(sc);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    rs[i] = b[i] - s * ax[i];
}

// keep the scaled warm start when s > 0 and |rs| < |b| (x = s x, r = rs), else x = 0, r = b
__global__ void k_warm_select(double* __restrict__ x, double* __restrict__ r, const double* __restrict__ b,
                              const double* __restrict__ rs, const double* __restrict__ sc, long long n) {
  lp_after_launch();
  const double s = lp_warm_scale(sc);
  const bool keep = s > 0.0 && sqrt(sc[7]) < sqrt(sc[0]);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    x[i] = keep ? x[i] * s : 0.0;
    r[i] = keep ? rs[i] : b[i];
  }
}

// The CG update split for fewer passes over the float64 fields: the step after A p only moves
// r (and its float32 copy) and forms |r|^2; x += alpha p is deferred to the pass that rebuilds p,
// which reads p anyway. alpha = rz / pap and beta = rz_new / rz are read on the device.
__global__ void k_cg_step_r(double* __restrict__ r, const double* __restrict__ ap, float* __restrict__ r32,
                            long long n, const double* __restrict__ num, const double* __restrict__ den,
                            double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  const double alpha = (*num) / (*den);
  double s = 0.0;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double ri = r[i] - alpha * ap[i];
    r[i] = ri;
    if (r32) r32[i] = (float)ri;
    s += ri * ri;
  }
  s = lp_block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// x += (rz / pap) p; p = z + (rz_new / rz) p
template <typename Tz>
__global__ void k_xpby_x(double* __restrict__ p, double* __restrict__ x, const Tz* __restrict__ z, long long n,
                         const double* __restrict__ rz, const double* __restrict__ pap,
                         const double* __restrict__ rz_new) {
  lp_after_launch();
  const double alpha = (*rz) / (*pap), beta = (*rz_new) / (*rz);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double pi = p[i];
    x[i] += alpha * pi;
    p[i] = (double)z[i] + beta * pi;
  }
}

}  // namespace

#define LP_GRID_ARGS int nx, int ny, int nz, int pz, int cpz
#define LP_GRID lp_grid(nx, ny, nz, pz, cpz)
#define LP_ST ((cudaStream_t)stream)
#define LP_VEC_GRID(n) lp_blocks((n), 256) > 148 * 32 ? 148 * 32 : lp_blocks((n), 256), 256, 0, LP_ST

namespace {
// a fine level and the level below it: on each axis the coarse cells are ceil(fine cells / 2),
// or one more when the coarse count is padded to even (loadpath/mg.py:607); the prolongation
// reads coarse nodes up to ceil(fine / 2), the restriction checks its fine reads against the fine
// grid
bool lp_axis_ok(int f, int c) { return c >= (f + 1) / 2 && c <= (f + 1) / 2 + 1; }
bool lp_pair_ok(const LpGrid& gf, const LpGrid& gc) {
  return lp_axis_ok(gf.nx, gc.nx) && lp_axis_ok(gf.ny, gc.ny) && lp_axis_ok(gf.nz, gc.nz);
}

template <typename T>
int launch_restrict(T* rc, T* d, const T* dinv, const double* coef, const T* b, const T* ax, const uint8_t* m,
                    const uint8_t* cm, const LpGrid& gf, const LpGrid& gc, int cols, cudaStream_t st) {
  if (!lp_grid_ok(gf) || !lp_grid_ok(gc) || !rc || !b || !ax || !m || !cm || cols < 1 || cols > 65535) return LP_ERR_ARG;
  if (d && (!dinv || !coef)) return LP_ERR_ARG;
  if (!lp_pair_ok(gf, gc)) return LP_ERR_ARG;
  const long long nw = (long long)((gc.NX() + R4_COLS - 1) / R4_COLS) * gc.NY() * (gc.pz / 4);
  lp_launch(k_restrict4<T>, dim3(lp_blocks(96 * nw, 128), cols), 128, 0, st, rc, d, dinv, coef, b, ax, m, cm, gf, gc);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

template <typename T>
int launch_prolong(T* x, const T* xc, const uint8_t* cm, const uint8_t* m, const LpGrid& gf, const LpGrid& gc, int cols,
                   cudaStream_t st) {
  if (!lp_grid_ok(gf) || !lp_grid_ok(gc) || !x || !xc || !m || !cm || cols < 1 || cols > 65535) return LP_ERR_ARG;
  if (!lp_pair_ok(gf, gc)) return LP_ERR_ARG;
  const long long t4 = gf.nodes_padded() / 4;
  // a component per thread while all three leave the GPU short of warps: to 64 x 32 x 32 cells (600 warps)
  // 2.3 us against 3.2, to 96 x 48 x 48 (1950) 4.1 against 3.8, to 256 x 128 x 128 43 against 27
  if (t4 / 32 * cols < 1500)
    lp_launch(k_prolong4<T, 1>, dim3(lp_blocks(t4, 128), 3, cols), 128, 0, st, x, xc, cm, m, gf, gc);
  else
    lp_launch(k_prolong4<T, 3>, dim3(lp_blocks(t4, 128), 1, cols), 128, 0, st, x, xc, cm, m, gf, gc);
  LP_LAUNCH_CHECK();
  return LP_OK;
}
}  // namespace

extern "C" {

int lpb_reduce_blocks(void) { return LP_RED_BLOCKS; }

// record a CUDA event on a stream; inside a stream capture it becomes an event-record node, so
// every replay of the graph records it again (for timing kernels inside graphs)
int lpb_event_record(void* event, void* stream) {
  if (!event) return LP_ERR_ARG;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(LP_ST, &cs) != cudaSuccess) return LP_ERR_LAUNCH;
  const cudaError_t e = cs == cudaStreamCaptureStatusActive
                            ? cudaEventRecordWithFlags((cudaEvent_t)event, LP_ST, cudaEventRecordExternal)
                            : cudaEventRecord((cudaEvent_t)event, LP_ST);
  return e == cudaSuccess ? LP_OK : LP_ERR_LAUNCH;
}

int lpb_dot_f64(const double* a, const double* b, long long n, double* part, double* out, void* stream) {
  if (!a || !b || !part || !out || n < 0) return LP_ERR_ARG;
  lp_launch(k_dot_partial<double, double>, LP_RED_BLOCKS, LP_RED_THREADS, 0, LP_ST, a, b, n, part);
  lp_launch(k_sum_final, 1, 1024, 0, LP_ST, part, LP_RED_BLOCKS, out);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_dot_f32(const float* a, const float* b, long long n, double* part, double* out, void* stream) {
  if (!a || !b || !part || !out || n < 0) return LP_ERR_ARG;
  lp_launch(k_dot_partial<float, float>, LP_RED_BLOCKS, LP_RED_THREADS, 0, LP_ST, a, b, n, part);
  lp_launch(k_sum_final, 1, 1024, 0, LP_ST, part, LP_RED_BLOCKS, out);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_dot_f64_f32(const double* a, const float* b, long long n, double* part, double* out, void* stream) {
  if (!a || !b || !part || !out || n < 0) return LP_ERR_ARG;
  lp_launch(k_dot_partial<double, float>, LP_RED_BLOCKS, LP_RED_THREADS, 0, LP_ST, a, b, n, part);
  lp_launch(k_sum_final, 1, 1024, 0, LP_ST, part, LP_RED_BLOCKS, out);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cg_step(double* x, double* r, const double* p, const double* ap, float* r32, long long n, const double* num,
                const double* den, double* part, double* rr, void* stream) {
  if (!x || !r || !p || !ap || !num || !den || !part || !rr) return LP_ERR_ARG;
  lp_launch(k_cg_step, LP_RED_BLOCKS, LP_RED_THREADS, 0, LP_ST, x, r, p, ap, r32, n, num, den, part);
  lp_launch(k_sum_final, 1, 1024, 0, LP_ST, part, LP_RED_BLOCKS, rr);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_xpby_f32(double* p, const float* z, long long n, const double* num, const double* den, void* stream) {
  if (!p || !z || !num || !den) return LP_ERR_ARG;
  lp_launch(k_xpby<float>, LP_VEC_GRID(n), p, z, n, num, den);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_xpby_f64(double* p, const double* z, long long n, const double* num, const double* den, void* stream) {
  if (!p || !z || !num || !den) return LP_ERR_ARG;
  lp_launch(k_xpby<double>, LP_VEC_GRID(n), p, z, n, num, den);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_axpby_f64(double* out, double a, const double* x, double b, const double* y, long long n, void* stream) {
  if (!out || !x) return LP_ERR_ARG;
  lp_launch(k_axpby<double>, LP_VEC_GRID(n), out, a, x, b, y, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_axpby_f32(float* out, float a, const float* x, float b, const float* y, long long n, void* stream) {
  if (!out || !x) return LP_ERR_ARG;
  lp_launch(k_axpby<float>, LP_VEC_GRID(n), out, a, x, b, y, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cast_f64_f32(float* out, const double* a, long long n, void* stream) {
  if (!out || !a) return LP_ERR_ARG;
  lp_launch(k_cast<double, float>, LP_VEC_GRID(n), out, a, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cast_f32_f64(double* out, const float* a, long long n, void* stream) {
  if (!out || !a) return LP_ERR_ARG;
  lp_launch(k_cast<float, double>, LP_VEC_GRID(n), out, a, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cheb_coef(double* coef, const double* vv, const double* vav, int its, int degree, double safety,
                  void* stream) {
  if (!coef || !vv || !vav || its < 1 || degree < 1 || degree > LP_CHEB_MAX_DEGREE) return LP_ERR_ARG;
  lp_launch(k_cheb_coef, 1, 1, 0, LP_ST, coef, vv, vav, its, degree, safety);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cheb_start_f32(const float* b, const float* dinv, const double* coef, float* x, float* r, float* d,
                       long long n, void* stream) {
  if (!b || !dinv || !coef || !x || !r || !d) return LP_ERR_ARG;
  lp_launch(k_cheb_start<float>, LP_VEC_GRID(n), b, dinv, coef, x, r, d, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cheb_start_f64(const double* b, const double* dinv, const double* coef, double* x, double* r, double* d,
                       long long n, void* stream) {
  if (!b || !dinv || !coef || !x || !r || !d) return LP_ERR_ARG;
  lp_launch(k_cheb_start<double>, LP_VEC_GRID(n), b, dinv, coef, x, r, d, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_residual_scaled_f32(const float* b, const float* ax, const float* dinv, const double* coef, float* r,
                            float* d, long long n, void* stream) {
  if (!b || !ax || !dinv || !coef || !r || !d) return LP_ERR_ARG;
  lp_launch(k_residual_scaled<float>, LP_VEC_GRID(n), b, ax, dinv, coef, r, d, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_residual_scaled_f64(const double* b, const double* ax, const double* dinv, const double* coef, double* r,
                            double* d, long long n, void* stream) {
  if (!b || !ax || !dinv || !coef || !r || !d) return LP_ERR_ARG;
  lp_launch(k_residual_scaled<double>, LP_VEC_GRID(n), b, ax, dinv, coef, r, d, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cheb_f32(float* x, float* d, float* r, const float* ad, const float* dinv, const double* coef, int step,
                 int last, long long n, void* stream) {
  if (!x || !d || !r || !ad || !dinv || !coef || step < 0 || step >= LP_CHEB_MAX_DEGREE) return LP_ERR_ARG;
  lp_launch(k_cheb<float>, LP_VEC_GRID(n), x, d, r, ad, dinv, coef, step, last, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_cheb_f64(double* x, double* d, double* r, const double* ad, const double* dinv, const double* coef, int step,
                 int last, long long n, void* stream) {
  if (!x || !d || !r || !ad || !dinv || !coef || step < 0 || step >= LP_CHEB_MAX_DEGREE) return LP_ERR_ARG;
  lp_launch(k_cheb<double>, LP_VEC_GRID(n), x, d, r, ad, dinv, coef, step, last, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

#define LP_CHEB2_ENTRIES(T, SFX)                                                                            \
  int lpb_cheb_d_start_##SFX(const T* b, const T* dinv, const double* coef, T* d, long long n, void* stream) { \
    if (!b || !dinv || !coef || !d) return LP_ERR_ARG;                                                   \
    lp_launch(k_cheb_d_start<T>, LP_VEC_GRID(n), b, dinv, coef, d, n);                                          \
    LP_LAUNCH_CHECK();                                                                                    \
    return LP_OK;                                                                                         \
  }                                                                                                       \
  int lpb_cheb2_zero_##SFX(T* x, const T* b, const T* ad, const T* d, const T* dinv, const double* coef,  \
                           long long n, void* stream) {                                                  \
    if (!x || !b || !ad || !d || !dinv || !coef) return LP_ERR_ARG;                                     \
    lp_launch(k_cheb2_zero<T>, LP_VEC_GRID(n), x, b, ad, d, dinv, coef, n);                                     \
    LP_LAUNCH_CHECK();                                                                                    \
    return LP_OK;                                                                                         \
  }                                                                                                       \
  int lpb_cheb2_##SFX(T* x, const T* d, const T* r, const T* ad, const T* dinv, const double* coef,       \
                      long long n, void* stream) {                                                       \
    if (!x || !d || !r || !ad || !dinv || !coef) return LP_ERR_ARG;                                     \
    lp_launch(k_cheb2<T>, LP_VEC_GRID(n), x, d, r, ad, dinv, coef, n);                                          \
    LP_LAUNCH_CHECK();                                                                                    \
    return LP_OK;                                                                                         \
  }
LP_CHEB2_ENTRIES(float, f32)
LP_CHEB2_ENTRIES(double, f64)

int lpb_cg_step_r(double* r, const double* ap, float* r32, long long n, const double* num, const double* den,
                  double* part, double* rr, void* stream) {
  if (!r || !ap || !num || !den || !part || !rr) return LP_ERR_ARG;
  lp_launch(k_cg_step_r, LP_RED_BLOCKS, LP_RED_THREADS, 0, LP_ST, r, ap, r32, n, num, den, part);
  lp_launch(k_sum_final, 1, 1024, 0, LP_ST, part, LP_RED_BLOCKS, rr);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_xpby_x_f32(double* p, double* x, const float* z, long long n, const double* rz, const double* pap,
                   const double* rz_new, void* stream) {
  if (!p || !x || !z || !rz || !pap || !rz_new) return LP_ERR_ARG;
  lp_launch(k_xpby_x<float>, LP_VEC_GRID(n), p, x, z, n, rz, pap, rz_new);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_xpby_x_f64(double* p, double* x, const double* z, long long n, const double* rz, const double* pap,
                   const double* rz_new, void* stream) {
  if (!p || !x || !z || !rz || !pap || !rz_new) return LP_ERR_ARG;
  lp_launch(k_xpby_x<double>, LP_VEC_GRID(n), p, x, z, n, rz, pap, rz_new);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_jacobi_f32(float* x, const float* b, const float* ax, const float* dinv, float omega, int from_zero,
                   long long n, void* stream) {
  lp_launch(k_jacobi<float>, LP_VEC_GRID(n), x, b, ax, dinv, omega, from_zero, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_jacobi_f64(double* x, const double* b, const double* ax, const double* dinv, double omega, int from_zero,
                   long long n, void* stream) {
  lp_launch(k_jacobi<double>, LP_VEC_GRID(n), x, b, ax, dinv, omega, from_zero, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

#define LP_FC_ARGS int fnx, int fny, int fnz, int fpz, int fcpz, int cnx, int cny, int cnz, int cpz_, int ccpz
#define LP_GF lp_grid(fnx, fny, fnz, fpz, fcpz)
#define LP_GC lp_grid(cnx, cny, cnz, cpz_, ccpz)

int lpb_restrict_residual_f32(float* rc, const float* b, const float* ax, const uint8_t* m, const uint8_t* cm,
                              LP_FC_ARGS, void* stream) {
  return launch_restrict<float>(rc, nullptr, nullptr, nullptr, b, ax, m, cm, LP_GF, LP_GC, 1, LP_ST);
}

// the same for cols columns (each field's columns one after the other), with the smoother's first
// direction on the coarse level, d = (dinv rc) coef[1] (d NULL: none)
int lpb_restrict_start_f32(float* rc, float* d, const float* dinv, const double* coef, const float* b, const float* ax,
                           const uint8_t* m, const uint8_t* cm, LP_FC_ARGS, int cols, void* stream) {
  return launch_restrict<float>(rc, d, dinv, coef, b, ax, m, cm, LP_GF, LP_GC, cols, LP_ST);
}

int lpb_restrict_residual_f64(double* rc, const double* b, const double* ax, const uint8_t* m, const uint8_t* cm,
                              LP_FC_ARGS, void* stream) {
  return launch_restrict<double>(rc, nullptr, nullptr, nullptr, b, ax, m, cm, LP_GF, LP_GC, 1, LP_ST);
}

// the same for cols columns (each field's columns one after the other), with the smoother's first
// direction on the coarse level, d = (dinv rc) coef[1] (d NULL: none)
int lpb_restrict_start_f64(double* rc, double* d, const double* dinv, const double* coef, const double* b, const double* ax,
                           const uint8_t* m, const uint8_t* cm, LP_FC_ARGS, int cols, void* stream) {
  return launch_restrict<double>(rc, d, dinv, coef, b, ax, m, cm, LP_GF, LP_GC, cols, LP_ST);
}

int lpb_prolong_add_f32(float* x, const float* xc, const uint8_t* cm, const uint8_t* m, LP_FC_ARGS, void* stream) {
  return launch_prolong<float>(x, xc, cm, m, LP_GF, LP_GC, 1, LP_ST);
}

// the same for cols columns
int lpb_prolong_add_cols_f32(float* x, const float* xc, const uint8_t* cm, const uint8_t* m, LP_FC_ARGS, int cols,
                             void* stream) {
  return launch_prolong<float>(x, xc, cm, m, LP_GF, LP_GC, cols, LP_ST);
}

int lpb_prolong_add_f64(double* x, const double* xc, const uint8_t* cm, const uint8_t* m, LP_FC_ARGS, void* stream) {
  return launch_prolong<double>(x, xc, cm, m, LP_GF, LP_GC, 1, LP_ST);
}

// the same for cols columns
int lpb_prolong_add_cols_f64(double* x, const double* xc, const uint8_t* cm, const uint8_t* m, LP_FC_ARGS, int cols,
                             void* stream) {
  return launch_prolong<double>(x, xc, cm, m, LP_GF, LP_GC, cols, LP_ST);
}

int lpb_mask_field_f32(float* out, const float* u, const uint8_t* m, LP_GRID_ARGS, int bitshift, void* stream) {
  LpGrid g = LP_GRID;
  long long n = 3 * g.nodes_padded();
  lp_launch(k_mask_field<float>, LP_VEC_GRID(n / 4), out, u, m, g, bitshift);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_mask_field_f64(double* out, const double* u, const uint8_t* m, LP_GRID_ARGS, int bitshift, void* stream) {
  LpGrid g = LP_GRID;
  long long n = 3 * g.nodes_padded();
  lp_launch(k_mask_field<double>, LP_VEC_GRID(n / 4), out, u, m, g, bitshift);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_scale_rsqrt_f32(float* v, long long n, const double* nrm2, void* stream) {
  lp_launch(k_scale_rsqrt<float>, LP_VEC_GRID(n), v, n, nrm2);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_scale_rsqrt_f64(double* v, long long n, const double* nrm2, void* stream) {
  lp_launch(k_scale_rsqrt<double>, LP_VEC_GRID(n), v, n, nrm2);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_dinv_mask_f32(float* av, const float* dinv, const uint8_t* m, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  long long n = 3 * g.nodes_padded();
  lp_launch(k_dinv_mask<float>, LP_VEC_GRID(n / 4), av, dinv, m, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_dinv_mask_f64(double* av, const double* dinv, const uint8_t* m, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  long long n = 3 * g.nodes_padded();
  lp_launch(k_dinv_mask<double>, LP_VEC_GRID(n / 4), av, dinv, m, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_warm_residual(double* rs, const double* b, const double* ax, const double* sc, long long n, void* stream) {
  if (!rs || !b || !ax || !sc || n < 0) return LP_ERR_ARG;
  lp_launch(k_warm_residual, LP_VEC_GRID(n), rs, b, ax, sc, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

int lpb_warm_select(double* x, double* r, const double* b, const double* rs, const double* sc, long long n,
                    void* stream) {
  if (!x || !r || !b || !rs || !sc || n < 0) return LP_ERR_ARG;
  lp_launch(k_warm_select, LP_VEC_GRID(n), x, r, b, rs, sc, n);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

}  // extern "C"
