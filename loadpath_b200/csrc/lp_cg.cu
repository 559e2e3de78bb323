// The PCG's and the power iteration's vector passes with their reductions folded into the pass that
// needs the result (loadpath/mg.py:771-794, :872-926). Each pass leaves one partial sum per block;
// the next pass's blocks all add those partials themselves, in the same order, so no launch
// of its own stands between a reduction and its use: with lpb_dot_*, lpb_cg_step_r and lpb_xpby_x_* an
// iteration took nine launches and a copy beside its V-cycle, with these five; a power step took seven
// beside its apply, with these one. The vectors stream with 16-byte accesses: at 256 x 128 x 128
// cells the passes over p, x and r are at the copy bandwidth, on the coarser grids a launch's 2 to 3 us is
// what counts.
//
// Every pass takes `cols` columns (right-hand sides): column j's fields start n values after
// column j - 1's, its scalars sc 8 doubles, its partials one row after. sc: [0] b.b, [1] r.z the
// step sizes use, [2] r.z newest, [3] p.Ap, [4] |r|^2.
#include "lp_common.cuh"

#define LP_ST ((cudaStream_t)stream)

namespace {

constexpr int CG_THREADS = 256;
constexpr int CG_BLOCKS = 592;   // 4 per SM on 148 SMs; also the most partials a pass leaves

// blocks of a pass over n values, four at a time (n / 4 of them)
inline int cg_blocks(long long n4) { return lp_blocks(n4, CG_THREADS) < CG_BLOCKS ? lp_blocks(n4, CG_THREADS) : CG_BLOCKS; }

// the sum of a pass's partials, the same bits in every block
__device__ __forceinline__ double part_sum(const double* __restrict__ part, int n, double* sh) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  return lp_block_sum(s, sh);
}
__device__ __forceinline__ double warp_part_sum(const double* __restrict__ part, int n) {
  double s = 0.0;
  for (int i = threadIdx.x & 31; i < n; i += 32) s += part[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// alpha = rz / p.Ap (p.Ap from the fine apply's partials); r -= alpha ap; r32 = (float)r; the
// smoother's first direction d = (dinv r) s; partials of |r|^2. sc[1] becomes the rz used here.
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
k_cg_r(double* __restrict__ r, const double* __restrict__ ap, float* __restrict__ r32, T* __restrict__ d,
       const T* __restrict__ dinv, const double* __restrict__ coef, long long n, double* __restrict__ sc,
       const double* __restrict__ pap_part, int npap, double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  const int col = blockIdx.y;
  const long long off = col * n;
  double* s = sc + 8 * col;
  const double pap = part_sum(pap_part + (long long)col * npap, npap, sh);
  const double rz = s[2], alpha = rz / pap;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    s[1] = rz;
    s[3] = pap;
  }
  const T sd = d ? (T)coef[1] : T(0);
  double acc = 0.0;
  for (long long i = 4 * (blockIdx.x * (long long)CG_THREADS + threadIdx.x); i < n; i += 4LL * gridDim.x * CG_THREADS) {
    double rv[4], av[4];
    lp_ld4(r + off + i, rv);
    lp_ld4(ap + off + i, av);
    float f[4];
    T t[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      rv[q] -= alpha * av[q];
      f[q] = (float)rv[q];
      acc += rv[q] * rv[q];
    }
    lp_st4(r + off + i, rv);
    if (r32) lp_st4(r32 + off + i, f);
    if (d) {
      lp_ld4(dinv + i, t);
#pragma unroll
      for (int q = 0; q < 4; ++q) t[q] = (t[q] * (T)rv[q]) * sd;
      lp_st4(d + off + i, t);
    }
  }
  acc = lp_block_sum(acc, sh);
  if (threadIdx.x == 0) part[(long long)col * gridDim.x + blockIdx.x] = acc;
}

// sc[4] = |r|^2 of every column (a warp each)
__global__ void k_cg_rr(double* __restrict__ sc, const double* __restrict__ part, int nparts, int cols) {
  lp_after_launch();
  for (int j = threadIdx.x >> 5; j < cols; j += blockDim.x >> 5) {
    const double rr = warp_part_sum(part + (long long)j * nparts, nparts);
    if ((threadIdx.x & 31) == 0) sc[8 * j + 4] = rr;
  }
}

// The stopping test on the device (loadpath/mg.py:872-926, as the host loop makes it) after every
// column's |r|^2: state (cols + 1, 2), row j the iteration at which column j stopped and its status
// (0 while it runs, 1 converged, 2 zero right-hand side, 3 p.Ap not positive), row cols the iteration
// count. The loop continues while a column runs and fewer than maxiter iterations ran.
__global__ void k_cg_test(cudaGraphConditionalHandle handle, double* __restrict__ sc, const double* __restrict__ part,
                          int nparts, long long* __restrict__ state, int cols, double rtol, long long maxiter) {
  lp_after_launch();
  const long long it = state[2 * cols] + 1;
  bool running = false;
  for (int j = threadIdx.x >> 5; j < cols; j += blockDim.x >> 5) {
    const double rr = warp_part_sum(part + (long long)j * nparts, nparts);
    if (threadIdx.x & 31) continue;
    double* s = sc + 8 * j;
    s[4] = rr;
    if (state[2 * j + 1] != 0) continue;
    const double bb = s[0], pap = s[3];
    long long status = 0;
    if (bb == 0.0) status = 2;
    else if (!(pap > 0.0)) status = 3;
    else if (sqrt(rr) <= rtol * sqrt(bb)) status = 1;
    if (status) {
      state[2 * j] = it;
      state[2 * j + 1] = status;
    } else {
      running = true;
    }
  }
  running = __syncthreads_or(running);   // and every thread has read the count
  if (threadIdx.x == 0) {
    state[2 * cols] = it;
    cudaGraphSetConditional(handle, (running && it < maxiter) ? 1u : 0u);
  }
}

// partials of r.z
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
k_cg_rz(const double* __restrict__ r, const T* __restrict__ z, long long n, double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  const long long off = blockIdx.y * n;
  double acc = 0.0;
  for (long long i = 4 * (blockIdx.x * (long long)CG_THREADS + threadIdx.x); i < n; i += 4LL * gridDim.x * CG_THREADS) {
    double rv[4];
    T zv[4];
    lp_ld4(r + off + i, rv);
    lp_ld4(z + off + i, zv);
#pragma unroll
    for (int q = 0; q < 4; ++q) acc += rv[q] * (double)zv[q];
  }
  acc = lp_block_sum(acc, sh);
  if (threadIdx.x == 0) part[(long long)blockIdx.y * gridDim.x + blockIdx.x] = acc;
}

// rz_new from k_cg_rz's partials; x += (rz / p.Ap) p; p = z + (rz_new / rz) p; sc[2] = rz_new
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
k_cg_p(double* __restrict__ p, double* __restrict__ x, const T* __restrict__ z, long long n, double* __restrict__ sc,
       const double* __restrict__ part, int nparts) {
  lp_after_launch();
  __shared__ double sh[32];
  const int col = blockIdx.y;
  const long long off = col * n;
  double* s = sc + 8 * col;
  const double rz_new = part_sum(part + (long long)col * nparts, nparts, sh);
  const double rz = s[1], alpha = rz / s[3], beta = rz_new / rz;
  if (blockIdx.x == 0 && threadIdx.x == 0) s[2] = rz_new;
  for (long long i = 4 * (blockIdx.x * (long long)CG_THREADS + threadIdx.x); i < n; i += 4LL * gridDim.x * CG_THREADS) {
    double pv[4], xv[4];
    T zv[4];
    lp_ld4(p + off + i, pv);
    lp_ld4(x + off + i, xv);
    lp_ld4(z + off + i, zv);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      xv[q] += alpha * pv[q];
      pv[q] = (double)zv[q] + beta * pv[q];
    }
    lp_st4(x + off + i, xv);
    lp_st4(p + off + i, pv);
  }
}

// ---- power iteration ---------------------------------------------------------------------------
// The vector is scaled one pass late: v' = m dinv (A v) / |v| from A of the unscaled v, the same
// iterate as normalising first, and v.v' / |v| the Rayleigh value of v / |v|. part: two rows of
// partials per step, |v'|^2 and v.v'.

// v = m v0; partials of |v|^2
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
k_pw_start(T* __restrict__ v, const T* __restrict__ v0, const uint8_t* __restrict__ m, LpGrid g, double* __restrict__ part) {
  lp_after_launch();
  __shared__ double sh[32];
  const long long nq = g.nodes_padded() >> 2;
  double acc = 0.0;
  for (long long i = blockIdx.x * (long long)CG_THREADS + threadIdx.x; i < 3 * nq; i += (long long)gridDim.x * CG_THREADS) {
    const int c = i >= nq ? (i >= 2 * nq ? 2 : 1) : 0;
    const unsigned mb = reinterpret_cast<const unsigned*>(m)[i - c * nq];
    T a[4];
    lp_ld4(v0 + 4 * i, a);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = ((mb >> (8 * q + c)) & 1) ? a[q] : T(0);
      acc += (double)a[q] * (double)a[q];
    }
    lp_st4(v + 4 * i, a);
  }
  acc = lp_block_sum(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// av = m dinv av / |v|; partials of |av|^2 and v.av; *vv = |v|^2
template <typename T>
__global__ void __launch_bounds__(CG_THREADS)
k_pw_step(T* __restrict__ av, const T* __restrict__ v, const T* __restrict__ dinv, const uint8_t* __restrict__ m,
          LpGrid g, const double* __restrict__ in, double* __restrict__ out, double* __restrict__ vv) {
  lp_after_launch();
  __shared__ double sh[32];
  const double s = part_sum(in, gridDim.x, sh);
  if (blockIdx.x == 0 && threadIdx.x == 0) *vv = s;
  const T nrm = s > 0.0 ? (T)sqrt(s) : T(1);
  const long long nq = g.nodes_padded() >> 2;
  double aa = 0.0, va = 0.0;
  for (long long i = blockIdx.x * (long long)CG_THREADS + threadIdx.x; i < 3 * nq; i += (long long)gridDim.x * CG_THREADS) {
    const int c = i >= nq ? (i >= 2 * nq ? 2 : 1) : 0;
    const unsigned mb = reinterpret_cast<const unsigned*>(m)[i - c * nq];
    T a[4], dv[4], u[4];
    lp_ld4(av + 4 * i, a);
    lp_ld4(dinv + 4 * i, dv);
    lp_ld4(v + 4 * i, u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      a[q] = ((mb >> (8 * q + c)) & 1) ? (dv[q] * a[q]) / nrm : T(0);
      aa += (double)a[q] * (double)a[q];
      va += (double)u[q] * (double)a[q];
    }
    lp_st4(av + 4 * i, a);
  }
  aa = lp_block_sum(aa, sh);
  va = lp_block_sum(va, sh);
  if (threadIdx.x == 0) {
    out[blockIdx.x] = aa;
    out[gridDim.x + blockIdx.x] = va;
  }
}

// lmax and the Chebyshev coefficients (k_cheb_coef's, from the last step's partials)
__global__ void k_pw_coef(double* __restrict__ coef, const double* __restrict__ vv, const double* __restrict__ part,
                          int nparts, int its, int degree, double safety) {
  lp_after_launch();
  const double va = warp_part_sum(part, nparts);
  if (threadIdx.x) return;
  bool zero = false;
  for (int k = 0; k < its; ++k) zero = zero || vv[k] == 0.0;
  const double lam = zero ? 0.0 : va / sqrt(vv[its - 1]);
  lp_cheb_coef(coef, lam, zero, degree, safety);
}

}  // namespace

extern "C" {

// the partials each pass of the entries below leaves for n values (a row of them per column)
int lpb_cg_parts(long long n) { return cg_blocks(n / 4); }

#define CG_ALIGNED(p) ((reinterpret_cast<uintptr_t>(p) & 15) == 0)

// r -= alpha ap (alpha = sc[2] / p.Ap, p.Ap the sum of npap partials), its float32 copy (may be
// NULL), the smoother's first direction d = (dinv r) coef[1] (d NULL: none); part: lpb_cg_parts(n)
// partials of |r|^2 per column; sc[1] = the r.z used, sc[3] = p.Ap. n a multiple of 4, fields on 16 bytes.
#define CG_R(T, SFX)                                                                                               \
  int lpb_cg_r_##SFX(double* r, const double* ap, float* r32, T* d, const T* dinv, const double* coef, long long n, \
                     double* sc, const double* pap_part, int npap, double* part, int cols, void* stream) {         \
    if (!r || !ap || !sc || !pap_part || !part || npap < 1 || cols < 1 || n < 4 || (n & 3)) return LP_ERR_ARG;     \
    if (d && (!dinv || !coef)) return LP_ERR_ARG;                                                                  \
    if (!CG_ALIGNED(r) || !CG_ALIGNED(ap) || !CG_ALIGNED(r32) || !CG_ALIGNED(d) || !CG_ALIGNED(dinv)) return LP_ERR_ARG; \
    lp_launch(k_cg_r<T>, dim3(cg_blocks(n / 4), cols), CG_THREADS, 0, LP_ST, r, ap, r32, d, dinv, coef, n, sc,     \
              pap_part, npap, part);                                                                               \
    LP_LAUNCH_CHECK();                                                                                             \
    return LP_OK;                                                                                                  \
  }
CG_R(float, f32)
CG_R(double, f64)

// sc[4] = |r|^2 of every column, from lpb_cg_r's partials
int lpb_cg_rr(double* sc, const double* part, long long n, int cols, void* stream) {
  if (!sc || !part || n < 4 || cols < 1) return LP_ERR_ARG;
  lp_launch(k_cg_rr, 1, 32 * (cols < 8 ? cols : 8), 0, LP_ST, sc, part, cg_blocks(n / 4), cols);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// the same, and the loop's stopping test (state (cols + 1, 2), zeroed before the loop) as one launch in
// the body of a device-side loop
int lpb_cg_test(long long handle, double* sc, const double* part, long long n, long long* state, int cols, double rtol,
                long long maxiter, void* stream) {
  if (!sc || !part || !state || n < 4 || cols < 1 || maxiter < 1) return LP_ERR_ARG;
  lp_launch(k_cg_test, 1, 32 * (cols < 8 ? cols : 8), 0, LP_ST, (cudaGraphConditionalHandle)handle, sc, part,
            cg_blocks(n / 4), state, cols, rtol, maxiter);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// part: lpb_cg_parts(n) partials of r.z per column; then lpb_cg_p: x += (sc[1] / sc[3]) p,
// p = z + (r.z / sc[1]) p, sc[2] = r.z
#define CG_RZ(T, SFX)                                                                                              \
  int lpb_cg_rz_##SFX(const double* r, const T* z, long long n, double* part, int cols, void* stream) {            \
    if (!r || !z || !part || n < 4 || (n & 3) || cols < 1 || !CG_ALIGNED(r) || !CG_ALIGNED(z)) return LP_ERR_ARG;  \
    lp_launch(k_cg_rz<T>, dim3(cg_blocks(n / 4), cols), CG_THREADS, 0, LP_ST, r, z, n, part);                      \
    LP_LAUNCH_CHECK();                                                                                             \
    return LP_OK;                                                                                                  \
  }                                                                                                                \
  int lpb_cg_p_##SFX(double* p, double* x, const T* z, long long n, double* sc, const double* part, int cols,      \
                     void* stream) {                                                                               \
    if (!p || !x || !z || !sc || !part || n < 4 || (n & 3) || cols < 1) return LP_ERR_ARG;                         \
    if (!CG_ALIGNED(p) || !CG_ALIGNED(x) || !CG_ALIGNED(z)) return LP_ERR_ARG;                                     \
    lp_launch(k_cg_p<T>, dim3(cg_blocks(n / 4), cols), CG_THREADS, 0, LP_ST, p, x, z, n, sc, part,                 \
              cg_blocks(n / 4));                                                                                   \
    LP_LAUNCH_CHECK();                                                                                             \
    return LP_OK;                                                                                                  \
  }
CG_RZ(float, f32)
CG_RZ(double, f64)

// Power iteration on D^-1 A: lpb_pw_start v = m v0; per step k, after av = A v, lpb_pw_step
// av = m dinv av / |v| and vv[k] = |v|^2, the two fields then trading places; lpb_pw_coef the
// Chebyshev coefficients after its steps. part: 4 * lpb_cg_parts(n) doubles; step: k, which selects the
// rows of partials. Fields on 16 bytes, the mask on 4.
#define PW(T, SFX)                                                                                                 \
  int lpb_pw_start_##SFX(T* v, const T* v0, const uint8_t* m, int nx, int ny, int nz, int pz, int cpz, double* part, \
                         void* stream) {                                                                           \
    const LpGrid g = lp_grid(nx, ny, nz, pz, cpz);                                                                 \
    if (!lp_grid_ok(g) || !v || !v0 || !m || !part || !CG_ALIGNED(v) || !CG_ALIGNED(v0)) return LP_ERR_ARG;        \
    const int nb = cg_blocks(3 * g.nodes_padded() / 4);                                                            \
    lp_launch(k_pw_start<T>, nb, CG_THREADS, 0, LP_ST, v, v0, m, g, part);                                         \
    LP_LAUNCH_CHECK();                                                                                             \
    return LP_OK;                                                                                                  \
  }                                                                                                                \
  int lpb_pw_step_##SFX(T* av, const T* v, const T* dinv, const uint8_t* m, int nx, int ny, int nz, int pz, int cpz, \
                        int step, double* part, double* vv, void* stream) {                                        \
    const LpGrid g = lp_grid(nx, ny, nz, pz, cpz);                                                                 \
    if (!lp_grid_ok(g) || !av || !v || !dinv || !m || !part || !vv || step < 0) return LP_ERR_ARG;                 \
    if (!CG_ALIGNED(av) || !CG_ALIGNED(v) || !CG_ALIGNED(dinv)) return LP_ERR_ARG;                                 \
    const int nb = cg_blocks(3 * g.nodes_padded() / 4);                                                            \
    lp_launch(k_pw_step<T>, nb, CG_THREADS, 0, LP_ST, av, v, dinv, m, g, part + 2 * nb * (step & 1),               \
              part + 2 * nb * (1 - (step & 1)), vv + step);                                                        \
    LP_LAUNCH_CHECK();                                                                                             \
    return LP_OK;                                                                                                  \
  }
PW(float, f32)
PW(double, f64)

int lpb_pw_coef(double* coef, const double* vv, const double* part, long long n, int its, int degree, double safety,
                void* stream) {
  if (!coef || !vv || !part || n < 4 || its < 1 || degree < 1 || degree > LP_CHEB_MAX_DEGREE) return LP_ERR_ARG;
  const int nb = cg_blocks(n / 4);
  lp_launch(k_pw_coef, 1, 32, 0, LP_ST, coef, vv, part + 2 * nb * (its & 1) + nb, nb, its, degree, safety);
  LP_LAUNCH_CHECK();
  return LP_OK;
}
}
