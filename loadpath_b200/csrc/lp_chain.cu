// The coarsest level's direct solve as a chain of node planes (loadpath/mg.py:708-754, where the
// reference calls SuperLU). The band (lp_band.cu) couples a plane of nodes, the slowest axis, only with
// its two neighbours, so separator planes cut it into segments that do not see one another:
//
//   A = [A_I  B; B^T  A_s],  A_I block diagonal over the segments, B sparse (27 entries per
//   separator dof and side), S = A_s - B^T A_I^-1 B block tridiagonal over the separators.
//
// What is stored: the dense inverse of every segment, W = A_I^-1 B of every segment (and its transpose)
// and the dense inverse of S. A solve is three matrix-vector passes that read each of them once:
//   y = A_I^-1 b_I, g = b_s - W^T b_I;   x_s = S^-1 g;   x_I = y - W x_s.
//
// Why. The band's factor and inverse are chains over all tile rows (one panel solve, product and pivot
// factor per 32 dofs, 9-10 us each) and the dense inverse of all n dofs is read whole by every solve:
// 411 MB at 31 x 11 x 7 nodes, 136 MB at 17 x 9 x 9. Here the segments are inverted side by side, so
// the chain is one segment's dofs and then the separators', and a solve reads 96 and 48 MB.
//
// Inverses are symmetric sweeps in place, 32 pivots at a time: with P = A_KK^-1 and Q = A_:K P,
//   A_KK <- -P,  A_:K <- Q,  A_rc <- A_rc - Q_r A_cK^T,
// after all of which A holds -A^-1; every step keeps the matrix symmetric, so only tiles on and
// below the diagonal are formed. A step is one launch over 64 x 64 tiles: the pivot's columns (the
// panel) and P come from buffers the launch before wrote, the launch writes the next panel as it
// goes, and one block forms and inverts the next pivot beside the others' updates.
//
// No pivoting, as the reference's symmetric mode. A sweep multiplies by inverses where the band's
// factor substitutes, so it is used only while every pivot keeps CHAIN_PIVOT_TOL of its original
// diagonal: a smaller, negative, zero or non-finite pivot is reported in *info and the caller takes
// the band's signed Cholesky instead (singular and roundoff-indefinite operators among them).
#include <algorithm>

#include "lp_common.cuh"
#include "lp_dmma.cuh"

namespace {

constexpr int CHAIN_MAX_SEG = 24;
constexpr int CHAIN_MAX_PLANE = 640;       // dofs of a plane
constexpr int CHAIN_COLS = 4;              // right-hand sides per pass of a solve
constexpr double CHAIN_PIVOT_TOL = 1e-9;
constexpr int CLD = 36;                    // shared row stride: each MMA operand load spreads over all banks

struct Chain {
  LpBand bd;
  int N0, b, P;                    // planes, dofs per plane, segments
  int start[CHAIN_MAX_SEG + 1];    // first plane of each segment; segment j ends before plane start[j + 1] - 1
  int M, MS, nS;                   // padded segment size, padded and real separator size
  // offsets in the workspace (doubles)
  long long ai, s, wt, w, el, er, diag, pan, pinv, y, g, xs, idx, total;
  __host__ __device__ int planes(int j) const { return start[j + 1] - 1 - start[j]; }
  __host__ __device__ int size(int j) const { return planes(j) * b; }
  __host__ __device__ int sep(int k) const { return start[k + 1] - 1; }   // plane of separator k
};

// Segment lengths: the P that minimizes the sweeps' steps in sequence, priced at 5 us each, plus their operations,
// at 12 TFLOP/s (measured, a step with its operations takes 11 us alone and 12 to 15 beside the power
// iterations); false when the band is the better form (too few planes to cut, or a plane
// or chain beyond the tables).
bool chain_plan(int nx, int ny, int nz, Chain& c) {
  c.bd = lp_band(nx + 1, ny + 1, nz + 1);
  const int ext[3] = {nx + 1, ny + 1, nz + 1};
  c.N0 = ext[c.bd.perm[0]];
  c.b = 3 * c.bd.N1 * c.bd.N2;
  if (c.N0 < 5 || c.b > CHAIN_MAX_PLANE || c.bd.n > (1 << 20)) return false;
  double best = 0.0;
  int bestP = 0;
  for (int P = 2; P <= CHAIN_MAX_SEG && 2 * P - 1 <= c.N0; ++P) {
    const int inner = c.N0 - (P - 1), len = (inner + P - 1) / P;
    const double m = (double)len * c.b, ms = (double)(P - 1) * c.b;
    const double t = 5e-6 * (m + ms) / 32.0 + (P * m * m * m + ms * ms * ms) / 12e12;
    if (!bestP || t < best) {
      best = t;
      bestP = P;
    }
  }
  c.P = bestP;
  const int inner = c.N0 - (c.P - 1);
  int p = 0, longest = 0;
  for (int j = 0; j < c.P; ++j) {
    const int len = inner / c.P + (j < inner % c.P ? 1 : 0);
    longest = std::max(longest, len);
    c.start[j] = p;
    p += len + 1;
  }
  c.start[c.P] = p;   // N0 + 1
  c.nS = (c.P - 1) * c.b;
  c.M = (longest * c.b + 63) / 64 * 64;
  c.MS = (c.nS + 63) / 64 * 64;
  long long o = 0;
  auto take = [&](long long n) {
    const long long at = o;
    o += (n + 15) / 16 * 16;
    return at;
  };
  const long long M = c.M, MS = c.MS, b = c.b, P = c.P;
  c.ai = take(P * M * M);
  c.s = take(MS * MS);
  c.wt = take(P * 2 * b * M);
  c.w = take(P * M * 2 * b);
  c.el = take(P * 27 * b);
  c.er = take(P * 27 * b);
  c.diag = take(P * M + MS);
  c.pan = take(2 * 32 * std::max(P * M, MS));
  c.pinv = take(2 * 1024 * P);
  c.y = take(CHAIN_COLS * 32LL * c.bd.nt);
  c.g = take(CHAIN_COLS * MS);
  c.xs = take(CHAIN_COLS * MS);
  c.idx = take((c.bd.n + 1) / 2);
  c.total = o;
  return true;
}

// entry (i, j) of the band
__device__ __forceinline__ double band_at(const double* __restrict__ t, const LpBand& bd, int i, int j) {
  if (i < j) {
    const int s = i;
    i = j;
    j = s;
  }
  const int R = i >> 5, d = R - (j >> 5);
  return d > bd.D ? 0.0 : __ldg(t + ((long long)R * (bd.D + 1) + d) * 1024 + (i & 31) * 32 + (j & 31));
}

// entry q of separator dof r's 27 couplings with a neighbouring plane: the dof of that plane, -1 past
// the plane's edge
__device__ __forceinline__ int couple_dof(const LpBand& bd, int r, int q) {
  const int node = r / 3, p1 = node / bd.N2 + q / 9 - 1, p2 = node % bd.N2 + (q / 3) % 3 - 1;
  return p1 < 0 || p2 < 0 || p1 >= bd.N1 || p2 >= bd.N2 ? -1 : 3 * (p1 * bd.N2 + p2) + q % 3;
}

// the segments' matrices (tiles on and below the diagonal; identity past a segment's dofs), the
// separators' couplings, the original diagonals and the dofs' places in a field
__global__ void k_chain_gather(double* __restrict__ ws, const double* __restrict__ t, Chain c, LpGrid g) {
  lp_after_launch();
  const long long M = c.M, na = c.P * M * M, ne = 2LL * (c.P - 1) * 27 * c.b, nd = c.P * M + c.MS;
  const long long total = na + ne + nd + c.bd.n;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    if (e < na) {
      const int j = (int)(e / (M * M)), q = (int)(e - j * M * M), i = q / c.M, k = q - i * c.M;
      if ((k >> 5) > (i >> 5)) continue;
      const int m = c.size(j), o = c.start[j] * c.b;
      ws[c.ai + e] = i < m && k < m ? band_at(t, c.bd, o + i, o + k) : (i == k ? 1.0 : 0.0);
    } else if (e < na + ne) {
      const long long f = e - na;
      const int r = (int)(f % c.b), q = (int)((f / c.b) % 27), ks = (int)(f / (27LL * c.b)), k = ks >> 1;
      const int p = c.sep(k), right = ks & 1, d = couple_dof(c.bd, r, q);
      const double v = d < 0 ? 0.0 : band_at(t, c.bd, p * c.b + r, (right ? p + 1 : p - 1) * c.b + d);
      ws[(right ? c.er : c.el) + (27LL * k + q) * c.b + r] = v;
    } else if (e < na + ne + nd) {
      const int f = (int)(e - na - ne);
      double v = 1.0;
      if (f < c.P * c.M) {
        const int j = f / c.M, i = f - j * c.M;
        if (i < c.size(j)) v = band_at(t, c.bd, c.start[j] * c.b + i, c.start[j] * c.b + i);
      } else if (f - c.P * c.M < c.nS) {
        const int i = f - c.P * c.M, k = i / c.b, d = c.sep(k) * c.b + i - k * c.b;
        v = band_at(t, c.bd, d, d);
      }
      ws[c.diag + f] = v;
    } else {
      const int i = (int)(e - na - ne - nd);
      int x, y, z;
      c.bd.coords(i / 3, x, y, z);
      reinterpret_cast<int*>(ws + c.idx)[i] = (int)((i % 3) * g.comp_stride() + g.node(x, y, z));
    }
  }
}

// 1 / d by the Newton-Raphson iteration for a reciprocal, x <- x + x (1 - d x), which squares the relative
// error: two steps from the hardware's approximation (20 bits) pass a double's 53. A pivot waits for it;
// d is a tested pivot, so the special cases that a division looks after do not arise (a zero, an infinity
// or a NaN gives a NaN that the caller's test reports).
__device__ __forceinline__ double pivot_inverse(double d) {
  double x;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
#pragma unroll
  for (int i = 0; i < 2; ++i) x = fma(x, fma(-d, x, 1.0), x);
  return x;
}

// The 32 x 32 matrix in s (row stride CLD) to its inverse in p (32 x 32), by warp 0: lane r holds row r
// and sweeps the pivots in order, two at a time (one inverse of their 2 x 2 block in the chain instead
// of two), the pivots' columns passed through shared memory; diag: the pivots' original diagonal
// entries, of which each must keep CHAIN_PIVOT_TOL. The row turns by two places a step, so the pivots'
// entries are always the first and the steps are one loop: unrolled, a single warp spent its time
// fetching instructions (30 us, against 4).
struct alignas(16) PivotCols {
  double v[2][2][32];
};
__device__ __forceinline__ void invert32(double (&s)[32][CLD], PivotCols& col, double* __restrict__ p,
                                         const double* __restrict__ diag, int row0, int* __restrict__ info) {
  const int lane = threadIdx.x & 31;
  double x[32];   // x[c]: entry (lane, (k + c) mod 32)
#pragma unroll
  for (int k = 0; k < 32; ++k) x[k] = s[lane][k];
  const double keep = CHAIN_PIVOT_TOL * diag[lane];
  int bad = 0;
  double d0 = __shfl_sync(0xffffffffu, x[0], 0), e = __shfl_sync(0xffffffffu, x[1], 0);
  double d1 = __shfl_sync(0xffffffffu, x[1], 1);
#pragma unroll 1
  for (int k = 0; k < 32; k += 2) {
    double *c0 = col.v[(k >> 1) & 1][0], *c1 = col.v[(k >> 1) & 1][1];
    c0[(lane - k) & 31] = x[0];
    c1[(lane - k) & 31] = x[1];
    __syncwarp();
    const double det = fma(d0, d1, -e * e), inv = pivot_inverse(det);
    // the pivots are d0 and det / d0 (a NaN fails either test)
    if (lane == k && !(d0 > keep && d0 < 1e300)) bad = row0 + k + 1;
    if (lane == k + 1 && !(det > keep * d0 && det < 1e300)) bad = row0 + k + 2;
    // rows outside the block: x_c - (f0 a_0c + f1 a_1c), (f0, f1) = (x_0, x_1) P, P the block's inverse; the
    // block's rows: P a_c, as 0 - (...) with the rows of -P. The next pivots' columns come first: they
    // are what the next step waits for.
    const bool in0 = lane == k, in1 = lane == k + 1, in = in0 || in1;
    const double u = in0 ? -1.0 : in1 ? 0.0 : x[0], w = in1 ? -1.0 : in0 ? 0.0 : x[1];
    const double f0 = inv * fma(u, d1, -w * e), f1 = inv * fma(w, d0, -u * e);
    const double n0 = fma(-f0, c0[2], fma(-f1, c1[2], in ? 0.0 : x[2]));
    const double n1 = fma(-f0, c0[3], fma(-f1, c1[3], in ? 0.0 : x[3]));
    d0 = __shfl_sync(0xffffffffu, n0, (k + 2) & 31);
    e = __shfl_sync(0xffffffffu, n1, (k + 2) & 31);
    d1 = __shfl_sync(0xffffffffu, n1, (k + 3) & 31);
    x[0] = n0;
    x[1] = n1;
#pragma unroll
    for (int c = 4; c < 32; c += 2) {
      const double2 a0 = *reinterpret_cast<const double2*>(c0 + c), a1 = *reinterpret_cast<const double2*>(c1 + c);
      x[c - 2] = fma(-f0, a0.x, fma(-f1, a1.x, in ? 0.0 : x[c]));
      x[c - 1] = fma(-f0, a0.y, fma(-f1, a1.y, in ? 0.0 : x[c + 1]));
    }
    x[30] = f0;
    x[31] = f1;
  }
  if (bad) atomicCAS(info, 0, bad);
#pragma unroll
  for (int k = 0; k < 32; k += 2) *reinterpret_cast<double2*>(p + lane * 32 + k) = make_double2(-x[k], -x[k + 1]);
}

// one matrix of a batch
struct SweepJob {
  double* a;             // matrices at stride astride, row stride ld
  long long astride;
  int ld, n;             // n: matrices
  double* pan;           // [2][n][ld][32]
  double* pinv;          // [2][n][32][32]
  const double* diag;    // [n][ld]
  int* info;
  short steps[CHAIN_MAX_SEG];
};

// the first panel and pivot of every matrix
__global__ void __launch_bounds__(256) k_sweep_first(SweepJob job) {
  lp_after_launch();
  __shared__ double s[32][CLD];
  __shared__ PivotCols col;
  const int j = blockIdx.y;
  const double* a = job.a + j * job.astride;
  if (blockIdx.x == 0) {
#pragma unroll
    for (int e = threadIdx.x; e < 1024; e += 256) {
      const int r = e >> 5, c = e & 31;
      s[r][c] = r >= c ? a[(long long)r * job.ld + c] : a[(long long)c * job.ld + r];
    }
    __syncthreads();
    if (threadIdx.x < 32) invert32(s, col, job.pinv + 1024LL * j, job.diag + (long long)j * job.ld, 0, job.info);
  } else {
    const int R = blockIdx.x;
    double* pan = job.pan + ((long long)j * job.ld + 32 * R) * 32;
    for (int e = threadIdx.x; e < 1024; e += 256) pan[e] = a[(32LL * R + (e >> 5)) * job.ld + (e & 31)];
  }
}

// d += A B^T for RB x 4 blocks of 8 x 8: A's rows from a0, B's from b0, 32 columns; an operand is read
// once for all the blocks that share it (one read of shared memory per product otherwise, which
// took as long as the products)
template <int RB>
__device__ __forceinline__ void block_product(double (&d)[RB][4][2], const double (*a)[CLD], int a0,
                                              const double (*b)[CLD], int b0) {
  const int l = threadIdx.x & 31, g = l >> 2, h = l & 3;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    double av[RB], bv[4];
#pragma unroll
    for (int r = 0; r < RB; ++r) av[r] = a[a0 + 8 * r + g][k + h];
#pragma unroll
    for (int c = 0; c < 4; ++c) bv[c] = b[b0 + 8 * c + g][k + h];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) dmma(d[r][c][0], d[r][c][1], av[r], bv[c]);
  }
}
// rows [r0, r0 + 8) of Q = pan P for a warp, from shared pan and P into shared Q
__device__ __forceinline__ void panel_product(double (*q)[CLD], const double (*pan)[CLD], const double (*p)[CLD], int r0) {
  const int l = threadIdx.x & 31, g = l >> 2, h = l & 3;
  double d[1][4][2] = {};
  block_product<1>(d, pan, r0, p, 0);
#pragma unroll
  for (int cb = 0; cb < 4; ++cb)
    *reinterpret_cast<double2*>(&q[r0 + g][8 * cb + 2 * h]) = make_double2(d[0][cb][0], d[0][cb][1]);
}

struct alignas(16) SweepSmem {
  double pi[64][CLD], pj[64][CLD], p[32][CLD], qi[64][CLD], qj[64][CLD];
};

// Step K of a batch's sweeps. Block 0 of a matrix: the next pivot; the others: 64 x 64 tiles (I, J),
// I >= J, eight warps of 16 x 32 entries each (a warp lies in one 32 x 32 tile).
__global__ void __launch_bounds__(256, 2) k_sweep_step(SweepJob job, int K) {
  lp_after_launch();
  extern __shared__ __align__(16) unsigned char sw_raw[];
  SweepSmem& sm = *reinterpret_cast<SweepSmem*>(sw_raw);
  __shared__ PivotCols col;
  const int j = blockIdx.y, steps = job.steps[j], ld = job.ld;
  if (K >= steps) return;
  double* a = job.a + j * job.astride;
  const long long pn = (long long)job.n * ld * 32;
  const double* pan = job.pan + (K & 1) * pn + (long long)j * ld * 32;
  double* pan_next = job.pan + ((K + 1) & 1) * pn + (long long)j * ld * 32;
  const double* p = job.pinv + ((K & 1) * job.n + j) * 1024LL;
  double* p_next = job.pinv + (((K + 1) & 1) * job.n + j) * 1024LL;
  const int tid = threadIdx.x, w = tid >> 5, l = tid & 31, g = l >> 2, h = l & 3;
  // every load of a block is issued before the first of them is waited for
  const int er = tid >> 4, ec = 2 * (tid & 15);   // this thread's pair of each 16 rows of 32
  double2 lp[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) lp[u] = __ldg(reinterpret_cast<const double2*>(p + (16 * u + er) * 32 + ec));
  if (blockIdx.x == 0) {
    if (K + 1 >= steps) return;
    const int r0 = 32 * (K + 1);
    double2 li[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) li[u] = __ldg(reinterpret_cast<const double2*>(pan + (r0 + 16LL * u + er) * 32 + ec));
    double old[2][2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int blk = 2 * w + k, r = 8 * (blk >> 2) + g, c = 8 * (blk & 3) + 2 * h;
#pragma unroll
      for (int i = 0; i < 2; ++i) old[k][i] = a[(long long)(r0 + max(r, c + i)) * ld + r0 + min(r, c + i)];
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      *reinterpret_cast<double2*>(&sm.p[16 * u + er][ec]) = lp[u];
      *reinterpret_cast<double2*>(&sm.pi[16 * u + er][ec]) = li[u];
    }
    __syncthreads();
    if (w < 4) panel_product(sm.qi, sm.pi, sm.p, 8 * w);
    __syncthreads();
    // A_(K+1,K+1) - Q A^T: sixteen 8 x 8 blocks, two per warp
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int blk = 2 * w + k, rb = 8 * (blk >> 2), cb = 8 * (blk & 3), r = rb + g, c = cb + 2 * h;
      double d0 = 0.0, d1 = 0.0;
#pragma unroll
      for (int kk = 0; kk < 32; kk += 4) dmma(d0, d1, sm.qi[rb + g][kk + h], sm.pi[cb + g][kk + h]);
      sm.pj[r][c] = old[k][0] - d0;
      sm.pj[r][c + 1] = old[k][1] - d1;
    }
    __syncthreads();
    if (w == 0)
      invert32(*reinterpret_cast<double(*)[32][CLD]>(&sm.pj[0]), col, p_next, job.diag + (long long)j * ld + r0, r0,
               job.info);
    return;
  }
  // tile (I, J) of the lower triangle
  int I = (int)((sqrtf(8.0f * (float)(blockIdx.x - 1) + 1.0f) - 1.0f) * 0.5f);
  while ((I + 1) * (I + 2) / 2 <= (int)blockIdx.x - 1) ++I;
  while (I * (I + 1) / 2 > (int)blockIdx.x - 1) --I;
  const int J = (int)blockIdx.x - 1 - I * (I + 1) / 2;
  if (2 * I >= steps) return;
  double2 li[4], lj[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    li[u] = __ldg(reinterpret_cast<const double2*>(pan + (64LL * I + 16 * u + er) * 32 + ec));
    lj[u] = __ldg(reinterpret_cast<const double2*>(pan + (64LL * J + 16 * u + er) * 32 + ec));
  }
  const int R = 2 * I + (w >> 2), C = 2 * J + (w & 1);
  const int lr = 16 * (w >> 1), lc = 32 * (w & 1);     // the warp's place in the 64 x 64 tile
  const int sr = lr & 31;                               // its first row in the 32 x 32 tile
  const bool update = R != K && C != K && R >= C && R < steps && !(R == C && R == K + 1);
  // the old entries are loaded while the panel's product is formed
  double v[2][4][2];
  if (update) {
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int cb = 0; cb < 4; ++cb) {
        const double2 o = *reinterpret_cast<const double2*>(a + (64LL * I + lr + 8 * rb + g) * ld + 64 * J + lc + 8 * cb + 2 * h);
        v[rb][cb][0] = o.x;
        v[rb][cb][1] = o.y;
      }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) *reinterpret_cast<double2*>(&sm.p[16 * u + er][ec]) = lp[u];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    *reinterpret_cast<double2*>(&sm.pi[16 * u + er][ec]) = li[u];
    *reinterpret_cast<double2*>(&sm.pj[16 * u + er][ec]) = lj[u];
  }
  __syncthreads();
  panel_product(sm.qi, sm.pi, sm.p, 8 * w);
  const bool krow = (K >> 1) == I;
  if (krow) panel_product(sm.qj, sm.pj, sm.p, 8 * w);
  __syncthreads();
  if (R < C || R >= steps || (R == C && R == K + 1)) return;
  if (update) {
    double d[2][4][2] = {};
    block_product<2>(d, sm.qi, lr, sm.pj, lc);
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int cb = 0; cb < 4; ++cb) {
        v[rb][cb][0] -= d[rb][cb][0];
        v[rb][cb][1] -= d[rb][cb][1];
      }
  } else {
#pragma unroll
    for (int rb = 0; rb < 2; ++rb)
#pragma unroll
      for (int cb = 0; cb < 4; ++cb) {
        const int tr = sr + 8 * rb + g, tc = 8 * cb + 2 * h;   // in the 32 x 32 tile
        const double* at = C != K ? nullptr : R == K ? &sm.p[tr][tc] : &sm.qi[lr + 8 * rb + g][tc];
        v[rb][cb][0] = at ? (R == K ? -at[0] : at[0]) : sm.qj[lc + tc][tr];
        v[rb][cb][1] = at ? (R == K ? -at[1] : at[1]) : sm.qj[lc + tc + 1][tr];
      }
  }
#pragma unroll
  for (int rb = 0; rb < 2; ++rb)
#pragma unroll
    for (int cb = 0; cb < 4; ++cb) {
      const int r = lr + 8 * rb + g, c = lc + 8 * cb + 2 * h;   // in the 64 x 64 tile
      const int tr = sr + 8 * rb + g, tc = 8 * cb + 2 * h;      // in the 32 x 32 tile
      const double o0 = v[rb][cb][0], o1 = v[rb][cb][1];
      *reinterpret_cast<double2*>(a + (64LL * I + r) * ld + 64 * J + c) = make_double2(o0, o1);
      if (C == K + 1) {
        *reinterpret_cast<double2*>(pan_next + (32LL * R + tr) * 32 + tc) = make_double2(o0, o1);
      } else if (R == K + 1) {
        pan_next[(32LL * C + tc) * 32 + tr] = o0;
        pan_next[(32LL * C + tc + 1) * 32 + tr] = o1;
      }
    }
}

// a <- -a, the lower triangle copied onto the upper, 32 x 32 tiles
__global__ void k_sweep_finish(double* __restrict__ a, long long astride, int ld) {
  lp_after_launch();
  __shared__ double s[32][33];
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bi < bj) return;
  a += blockIdx.z * astride;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;   // 32 x 8 threads
  for (int r = ty; r < 32; r += 8) {
    double* e = a + (32LL * bi + r) * ld + 32 * bj + tx;
    s[r][tx] = -*e;
    if (bi > bj || tx <= r) *e = s[r][tx];
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8)
    if (bi > bj || tx > r) a[(32LL * bj + r) * ld + 32 * bi + tx] = s[tx][r];
}

// W^T (2b x M per segment: the left separator's dofs, then the right one's) and W: a 32 x 32 tile of
// separator dofs and segment dofs per block
__global__ void __launch_bounds__(256) k_chain_w(double* __restrict__ ws, Chain c) {
  lp_after_launch();
  __shared__ double s[32][33];
  __shared__ double ec[32][27];
  __shared__ int dc[32][27];
  const int j = blockIdx.z >> 1, side = blockIdx.z & 1;   // side 0: separator j - 1, 1: separator j
  const int k = side ? j : j - 1;
  const int i0 = 32 * blockIdx.x, c0 = 32 * blockIdx.y, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int m = c.size(j);
  if (i0 >= m) return;
  if (k < 0 || k >= c.P - 1) {   // the chain's ends: no separator, columns of zeros (a solve reads them)
    for (int r = w; r < 32; r += 8)
      if (i0 + r < m && c0 + lane < c.b) ws[c.w + ((long long)j * c.M + i0 + r) * 2 * c.b + side * c.b + c0 + lane] = 0.0;
    return;
  }
  const double* ai = ws + c.ai + (long long)j * c.M * c.M;
  const double* e = ws + (side ? c.el : c.er) + 27LL * k * c.b;   // separator k and this segment's plane beside it
  const int po = side ? (c.planes(j) - 1) * c.b : 0;
  const int i = i0 + lane;
  for (int t = threadIdx.x; t < 32 * 27; t += 256) {   // the tile's couplings; a missing one weighs zero
    const int cl = t / 27, q = t - 27 * cl, cc = c0 + cl, d = cc < c.b ? couple_dof(c.bd, cc, q) : -1;
    ec[cl][q] = d < 0 ? 0.0 : __ldg(e + q * c.b + cc);
    dc[cl][q] = po + (d < 0 ? 0 : d);
  }
  __syncthreads();
  for (int q8 = 0; q8 < 4; ++q8) {
    const int cl = w + 8 * q8, cc = c0 + cl;
    double v = 0.0;
    if (cc < c.b) {
#pragma unroll
      for (int q = 0; q < 27; ++q) v += ec[cl][q] * __ldg(ai + (long long)dc[cl][q] * c.M + i);
      ws[c.wt + ((2LL * j + side) * c.b + cc) * c.M + i] = i < m ? v : 0.0;
    }
    s[w + 8 * q8][lane] = v;
  }
  __syncthreads();
  for (int r = w; r < 32; r += 8)
    if (i0 + r < m && c0 + lane < c.b) ws[c.w + ((long long)j * c.M + i0 + r) * 2 * c.b + side * c.b + c0 + lane] = s[lane][r];
}

// S = A_s - B^T W, tiles on and below the diagonal (identity past its dofs)
__global__ void __launch_bounds__(256) k_chain_schur(double* __restrict__ ws, const double* __restrict__ t, Chain c) {
  lp_after_launch();
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bi < bj) return;
  // the couplings of the tile's rows with the planes left and right of their separator
  __shared__ double el[32][27], er[32][27];
  __shared__ int dc[32][27];
  for (int e = threadIdx.x; e < 32 * 27; e += 256) {
    const int rl = e / 27, q = e - 27 * rl, ri = 32 * bi + rl, k = ri / c.b, r = ri - k * c.b;
    const int d = ri < c.nS ? couple_dof(c.bd, r, q) : -1;
    el[rl][q] = d < 0 ? 0.0 : ws[c.el + (27LL * k + q) * c.b + r];
    er[rl][q] = d < 0 ? 0.0 : ws[c.er + (27LL * k + q) * c.b + r];
    dc[rl][q] = d < 0 ? 0 : d;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int rl = threadIdx.x >> 5; rl < 32; rl += 8) {
    const int ri = 32 * bi + rl, rj = 32 * bj + lane;
    double v = ri == rj ? 1.0 : 0.0;
    if (ri < c.nS && rj < c.nS) {
      const int k = ri / c.b, r = ri - k * c.b, k2 = rj / c.b, cc = rj - k2 * c.b;
      v = 0.0;
      if (k == k2) {
        const int p = c.sep(k) * c.b;
        v = band_at(t, c.bd, p + r, p + cc);
        // through the last plane of the segment left of the separator (W's right columns) and the first
        // of the one right of it (its left columns)
        const double* wl = ws + c.w + ((long long)k * c.M + (c.planes(k) - 1) * c.b) * 2 * c.b + c.b + cc;
        const double* wr = ws + c.w + (long long)(k + 1) * c.M * 2 * c.b + cc;
#pragma unroll 9
        for (int q = 0; q < 27; ++q) {
          v -= el[rl][q] * wl[2LL * c.b * dc[rl][q]];
          v -= er[rl][q] * wr[2LL * c.b * dc[rl][q]];
        }
      } else if (k == k2 + 1) {
        const double* wl = ws + c.w + ((long long)k * c.M + (c.planes(k) - 1) * c.b) * 2 * c.b + cc;
#pragma unroll 9
        for (int q = 0; q < 27; ++q) v -= el[rl][q] * wl[2LL * c.b * dc[rl][q]];
      }
    }
    if (ri >= rj) ws[c.s + (long long)ri * c.MS + rj] = v;
  }
}

// ---- solve ---------------------------------------------------------------------------------
// A warp takes one row of a matrix. Its first loads are issued before the vector is staged in shared
// memory (they do not depend on the pass before), and eight 16-byte loads per lane are in flight at a
// time: a pass moves its matrix at the rate that the loads in flight allow.
constexpr int ROW_AHEAD = 8;
struct RowAhead {
  double2 x[ROW_AHEAD];
  template <bool EARLY = false>   // EARLY: before lp_wait_prior
  __device__ __forceinline__ void load(const double* __restrict__ a, int k0, int n) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < ROW_AHEAD; ++u) {
      const int k = k0 + 64 * u + 2 * lane;
      const double2* p = reinterpret_cast<const double2*>(a + k);
      x[u] = k < n ? (EARLY ? __ldcg(p) : __ldg(p)) : make_double2(0.0, 0.0);
    }
  }
  // s[c] += row . v_c over the loaded entries (v_c: NC shared vectors at stride vs); n even
  template <int NC>
  __device__ __forceinline__ void add(const double* v, int vs, int k0, int n, double (&s)[NC]) const {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int u = 0; u < ROW_AHEAD; ++u) {
      const int k = k0 + 64 * u + 2 * lane;
      if (k < n) {
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const double2 w = *reinterpret_cast<const double2*>(v + c * vs + k);
          s[c] += x[u].x * w.x;
          s[c] += x[u].y * w.y;
        }
      }
    }
  }
};
template <int NC>
__device__ __forceinline__ void row_dot(RowAhead& h, const double* __restrict__ a, int n, const double* v, int vs,
                                        double (&s)[NC]) {
  h.add<NC>(v, vs, 0, n, s);
  for (int k0 = 64 * ROW_AHEAD; k0 < n; k0 += 64 * ROW_AHEAD) {
    h.load(a, k0, n);
    h.add<NC>(v, vs, k0, n, s);
  }
}
template <int NC>
__device__ __forceinline__ void lane_sums(double (&s)[NC]) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_xor_sync(0xffffffffu, s[c], o);
}

constexpr int SOLVE_ROWS = 8;   // rows per block, one per warp
constexpr int SEG_ROWS = 16;    // rows of a segment's inverse per block, two per warp: half as many blocks stage b

// nothing: behind the factor's launches, so that they are complete for whatever is launched next, started
// early or not
__global__ void k_chain_settled() { lp_after_launch(); }

// rows of y = A_I^-1 b_I (blocks of each segment in turn), then of g = b_s - W^T b_I
template <typename T, int NC>
__global__ void __launch_bounds__(256) k_chain_y(double* __restrict__ ws, const T* __restrict__ f, long long cstride,
                                                 Chain c) {
  extern __shared__ __align__(16) unsigned char sv_raw[];
  double* v = reinterpret_cast<double*>(sv_raw);   // [2][NC][M]
  const int* idx = reinterpret_cast<const int*>(ws + c.idx);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto stage = [&](double* d, int j) {   // segment j's right-hand side, zero to M
    const int m = c.size(j), o = c.start[j] * c.b;
    for (int i = threadIdx.x; i < c.M; i += 256) {
      const int at = i < m ? idx[o + i] : 0;
#pragma unroll
      for (int q = 0; q < NC; ++q) d[q * c.M + i] = i < m ? (double)f[q * cstride + at] : 0.0;
    }
  };
  int blk = blockIdx.x;
  for (int j = 0; j < c.P; ++j) {
    const int m = c.size(j), nb = (m + SEG_ROWS - 1) / SEG_ROWS;
    if (blk >= nb) {
      blk -= nb;
      continue;
    }
    const int r = SEG_ROWS * blk + 2 * w, n = (m + 1) & ~1;
    const double* a0 = ws + c.ai + ((long long)j * c.M + min(r, m - 1)) * c.M;
    const double* a1 = ws + c.ai + ((long long)j * c.M + min(r + 1, m - 1)) * c.M;
    RowAhead h0, h1;
    h0.load<true>(a0, 0, n);
    h1.load<true>(a1, 0, n);   // (the matrices are older than the launch ahead: lpb_chain_factor sees to it)
    lp_after_launch();
    stage(v, j);
    __syncthreads();
    if (r >= m) return;
    double s0[NC] = {}, s1[NC] = {};
    row_dot<NC>(h0, a0, n, v, c.M, s0);
    row_dot<NC>(h1, a1, n, v, c.M, s1);
    lane_sums<NC>(s0);
    lane_sums<NC>(s1);
#pragma unroll
    for (int q = 0; q < NC; ++q)
      if (lane == q) {
        double* y = ws + c.y + q * 32LL * c.bd.nt + c.start[j] * c.b + r;
        y[0] = s0[q];
        if (r + 1 < m) y[1] = s1[q];
      }
    return;
  }
  const int nb = (c.b + SOLVE_ROWS - 1) / SOLVE_ROWS, k = blk / nb;   // separator
  const int r = SOLVE_ROWS * (blk - k * nb) + w, rr = min(r, c.b - 1);
  const double* wl = ws + c.wt + ((2LL * k + 1) * c.b + rr) * c.M;       // segment k, its right separator
  const double* wr = ws + c.wt + (2LL * (k + 1) * c.b + rr) * c.M;       // segment k + 1, its left separator
  const int nl = (c.size(k) + 1) & ~1, nr = (c.size(k + 1) + 1) & ~1;
  RowAhead hl, hr;
  hl.load<true>(wl, 0, nl);
  hr.load<true>(wr, 0, nr);
  lp_after_launch();
  stage(v, k);
  stage(v + NC * c.M, k + 1);
  __syncthreads();
  if (r >= c.b) return;
  double s[NC] = {};
  row_dot<NC>(hl, wl, nl, v, c.M, s);
  row_dot<NC>(hr, wr, nr, v + NC * c.M, c.M, s);
  lane_sums<NC>(s);
#pragma unroll
  for (int q = 0; q < NC; ++q)
    if (lane == q) ws[c.g + q * (long long)c.MS + k * c.b + r] = (double)f[q * cstride + idx[c.sep(k) * c.b + r]] - s[q];
}

// x_s = S^-1 g
template <typename T, int NC>
__global__ void __launch_bounds__(256) k_chain_s(double* __restrict__ ws, T* __restrict__ f, long long cstride, Chain c) {
  extern __shared__ __align__(16) unsigned char sv_raw[];
  double* v = reinterpret_cast<double*>(sv_raw);   // [NC][MS]
  const int* idx = reinterpret_cast<const int*>(ws + c.idx);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = SOLVE_ROWS * blockIdx.x + w, n = (c.nS + 1) & ~1;
  const double* a = ws + c.s + (long long)min(r, c.nS - 1) * c.MS;
  RowAhead h;
  h.load<true>(a, 0, n);   // (the matrix was complete before the launch ahead, k_chain_y)
  lp_wait_prior();
  lp_release_next();
#pragma unroll
  for (int q = 0; q < NC; ++q)
    for (int i = threadIdx.x; i < c.MS; i += 256) v[q * c.MS + i] = i < c.nS ? ws[c.g + q * (long long)c.MS + i] : 0.0;
  __syncthreads();
  if (r >= c.nS) return;
  double s[NC] = {};
  row_dot<NC>(h, a, n, v, c.MS, s);
  lane_sums<NC>(s);
#pragma unroll
  for (int q = 0; q < NC; ++q)
    if (lane == q) {
      ws[c.xs + q * (long long)c.MS + r] = s[q];
      f[q * cstride + idx[c.sep(r / c.b) * c.b + r % c.b]] = (T)s[q];
    }
}

// x_I = y - W x_s
template <typename T, int NC>
__global__ void __launch_bounds__(256) k_chain_x(double* __restrict__ ws, T* __restrict__ f, long long cstride, Chain c) {
  extern __shared__ __align__(16) unsigned char sv_raw[];
  double* v = reinterpret_cast<double*>(sv_raw);   // [NC][2b]: the segment's left and right separator
  const int* idx = reinterpret_cast<const int*>(ws + c.idx);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int blk = blockIdx.x, j = 0;
  for (; j < c.P; ++j) {
    const int nb = (c.size(j) + SOLVE_ROWS - 1) / SOLVE_ROWS;
    if (blk < nb) break;
    blk -= nb;
  }
  const int m = c.size(j), lo = j > 0 ? 0 : c.b, hi = j < c.P - 1 ? 2 * c.b : c.b;   // the columns there are
  const int r = SOLVE_ROWS * blk + w, n = 2 * c.b;
  const double* a = ws + c.w + ((long long)j * c.M + min(r, m - 1)) * n;
  RowAhead h;
  h.load<true>(a, 0, n);
  lp_wait_prior();
  lp_release_next();
#pragma unroll
  for (int q = 0; q < NC; ++q)
    for (int k = threadIdx.x; k < n; k += 256)
      v[q * n + k] = k >= lo && k < hi ? ws[c.xs + q * (long long)c.MS + (j - 1) * c.b + k] : 0.0;
  __syncthreads();
  if (r >= m) return;
  double s[NC] = {};
  row_dot<NC>(h, a, n, v, n, s);
  lane_sums<NC>(s);
#pragma unroll
  for (int q = 0; q < NC; ++q)
    if (lane == q) {
      const int i = c.start[j] * c.b + r;
      f[q * cstride + idx[i]] = (T)(ws[c.y + q * 32LL * c.bd.nt + i] - s[q]);
    }
}

int sweep_all(SweepJob job, cudaStream_t st) {
  int steps = 0;
  for (int j = 0; j < job.n; ++j) steps = std::max(steps, (int)job.steps[j]);
  const int smem = (int)sizeof(SweepSmem);
  if (cudaFuncSetAttribute(k_sweep_step, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
    return LP_ERR_LAUNCH;
  lp_launch(k_sweep_first, dim3((unsigned)(job.ld / 32), (unsigned)job.n), 256, 0, st, job);
  const int T = (steps + 1) / 2;
  for (int K = 0; K < steps; ++K)
    lp_launch(k_sweep_step, dim3((unsigned)(1 + T * (T + 1) / 2), (unsigned)job.n), 256, smem, st, job, K);
  const unsigned nt = (unsigned)(job.ld / 32);
  lp_launch(k_sweep_finish, dim3(nt, nt, (unsigned)job.n), 256, 0, st, job.a, job.astride, job.ld);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

template <typename T, int NC>
int chain_pass(double* ws, const T* fi, T* fo, long long cstride, const Chain& c, cudaStream_t st) {
  int rows = 0, pairs = 0;
  for (int j = 0; j < c.P; ++j) {
    rows += (c.size(j) + SOLVE_ROWS - 1) / SOLVE_ROWS;
    pairs += (c.size(j) + SEG_ROWS - 1) / SEG_ROWS;
  }
  const int gb = (c.P - 1) * ((c.b + SOLVE_ROWS - 1) / SOLVE_ROWS);
  const int s1 = 2 * NC * c.M * 8, s2 = NC * c.MS * 8, s3 = NC * 2 * c.b * 8;
  if (!lp_smem_limit((const void*)k_chain_y<T, NC>, s1) || !lp_smem_limit((const void*)k_chain_s<T, NC>, s2) ||
      !lp_smem_limit((const void*)k_chain_x<T, NC>, s3))
    return LP_ERR_SIZE;
  lp_launch(k_chain_y<T, NC>, pairs + gb, 256, s1, st, ws, fi, cstride, c);
  lp_launch(k_chain_s<T, NC>, (c.nS + SOLVE_ROWS - 1) / SOLVE_ROWS, 256, s2, st, ws, fo, cstride, c);
  lp_launch(k_chain_x<T, NC>, rows, 256, s3, st, ws, fo, cstride, c);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

template <typename T>
int chain_solve(T* fo, const T* fi, long long cstride, int ncol, double* ws, LpGrid g, cudaStream_t st) {
  Chain c;
  if (!lp_grid_ok(g) || !fo || !fi || !ws || ncol < 1 || (ncol > 1 && cstride < 3 * g.comp_stride()) ||
      !chain_plan(g.nx, g.ny, g.nz, c))
    return LP_ERR_ARG;
  // as many columns per pass as their vectors fit in shared memory beside one another
  const long long need = 8LL * std::max(2 * c.M, c.MS);
  int most = CHAIN_COLS;
  while (most > 1 && most * need > 200 * 1024) most >>= 1;
  for (int q = 0; q < ncol;) {
    int n = std::min(most, ncol - q);
    if (n == 3) n = 2;
    const T* i = fi + q * cstride;
    T* o = fo + q * cstride;
    const int rc = n == 4 ? chain_pass<T, 4>(ws, i, o, cstride, c, st)
                   : n == 2 ? chain_pass<T, 2>(ws, i, o, cstride, c, st)
                            : chain_pass<T, 1>(ws, i, o, cstride, c, st);
    if (rc != LP_OK) return rc;
    q += n;
  }
  return LP_OK;
}

}  // namespace

#define LP_GRID_ARGS int nx, int ny, int nz, int pz, int cpz
#define LP_GRID lp_grid(nx, ny, nz, pz, cpz)
#define LP_ST ((cudaStream_t)stream)

extern "C" {

// doubles of workspace the chain form of a coarsest level takes, 0 where the band form is the one to use;
// out (may be NULL): segments, dofs per plane, padded segment size, separator dofs, kernels that
// lpb_chain_factor launches
long long lpb_chain_dims(int nx, int ny, int nz, long long* out) {
  Chain c;
  if (nx < 1 || ny < 1 || nz < 1 || !chain_plan(nx, ny, nz, c)) return 0;
  if (2LL * c.M * 8 > 220 * 1024 || c.MS * 8LL > 220 * 1024) return 0;
  if (out) {
    out[0] = c.P;
    out[1] = c.b;
    out[2] = c.M;
    out[3] = c.nS;
    out[4] = 8 + (c.size(0) + 31) / 32 + (c.nS + 31) / 32;
  }
  return c.total;
}

// The chain's inverses from the band t (lpb_coarse_band_*, not changed) into ws (lpb_chain_dims
// doubles, 16-byte aligned); *info (one device int, zeroed here): 0, or nonzero when a pivot lost its
// digits or its sign, and the level is to be factored as a band instead.
int lpb_chain_factor(double* ws, const double* t, int* info, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  Chain c;
  if (!lp_grid_ok(g) || !ws || (reinterpret_cast<uintptr_t>(ws) & 15) || !t || !info || !lpb_chain_dims(nx, ny, nz, nullptr) ||
      !chain_plan(nx, ny, nz, c))
    return LP_ERR_ARG;
  if (cudaMemsetAsync(info, 0, sizeof(int), LP_ST) != cudaSuccess) return LP_ERR_LAUNCH;
  lp_launch(k_chain_gather, 148 * 8, 256, 0, LP_ST, ws, t, c, g);
  SweepJob job{};
  job.a = ws + c.ai;
  job.astride = (long long)c.M * c.M;
  job.ld = c.M;
  job.n = c.P;
  job.pan = ws + c.pan;
  job.pinv = ws + c.pinv;
  job.diag = ws + c.diag;
  job.info = info;
  for (int j = 0; j < c.P; ++j) job.steps[j] = (short)((c.size(j) + 31) / 32);
  int rc = sweep_all(job, LP_ST);
  if (rc != LP_OK) return rc;
  lp_launch(k_chain_w, dim3((unsigned)(c.M / 32), (unsigned)((c.b + 31) / 32), (unsigned)(2 * c.P)), 256, 0, LP_ST, ws, c);
  lp_launch(k_chain_schur, dim3((unsigned)(c.MS / 32), (unsigned)(c.MS / 32)), 256, 0, LP_ST, ws, t, c);
  job.a = ws + c.s;
  job.astride = 0;
  job.ld = c.MS;
  job.n = 1;
  job.diag = ws + c.diag + (long long)c.P * c.M;
  job.steps[0] = (short)((c.nS + 31) / 32);
  rc = sweep_all(job, LP_ST);
  if (rc != LP_OK) return rc;
  lp_launch(k_chain_settled, 1, 32, 0, LP_ST);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// f_out = A^-1 f_in on the coarsest level from lpb_chain_factor's ws (whose solve scratch it uses: solves
// of one ws do not overlap)
int lpb_chain_solve_f32(float* f_out, const float* f_in, double* ws, LP_GRID_ARGS, void* stream) {
  return chain_solve<float>(f_out, f_in, 0, 1, ws, LP_GRID, LP_ST);
}

int lpb_chain_solve_f64(double* f_out, const double* f_in, double* ws, LP_GRID_ARGS, void* stream) {
  return chain_solve<double>(f_out, f_in, 0, 1, ws, LP_GRID, LP_ST);
}

// ncol right-hand sides: column c of f_in / f_out at element offset c * cstride (whole node fields)
int lpb_chain_solve_cols_f32(float* f_out, const float* f_in, long long cstride, int ncol, double* ws, LP_GRID_ARGS,
                             void* stream) {
  return chain_solve<float>(f_out, f_in, cstride, ncol, ws, LP_GRID, LP_ST);
}

int lpb_chain_solve_cols_f64(double* f_out, const double* f_in, long long cstride, int ncol, double* ws, LP_GRID_ARGS,
                             void* stream) {
  return chain_solve<double>(f_out, f_in, cstride, ncol, ws, LP_GRID, LP_ST);
}

}  // extern "C"
