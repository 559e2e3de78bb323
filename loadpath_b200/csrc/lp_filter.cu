// The cone density filter and its transpose (loadpath/simp.py:1143-1228,
// loadpath/benchmarks/reference.py:48-71), and loadpath's volume-multiplier trial that runs through
// it (loadpath/simp.py:2320-2376): OC step, filter, projection and projected volume in one pass.
// All in float64.
//
// What bounds it. Gathered tap by tap a cell costs one read of shared memory and one FMA per tap (27 taps
// at r = 2, 93 at r = 3) and several times that in address, branch and weight instructions: the
// instructions come first, shared memory and FP64 issue next, HBM (16-24 bytes a cell) last. The cone
// is symmetric, so the taps are taken by classes: the columns (dx, dy) with one dx^2 + dy^2 share
// their weights, so a thread adds up a class's staged columns of four z cells (two 16-byte reads and four
// additions a column) and then adds each listed w(class, |dz|) times those sums to the 4 + 2R cells
// they reach in z, kept in registers from one z chunk to the next: 25 reads of a column and 49
// operations a cell at r = 3, at constant offsets, and only the chunk in hand has to be staged.
//
// Work layout. A block takes 32 x 16 cell columns (lanes along x, a row per warp) and marches z over a
// segment, one chunk of four cells at a time, from the chunk below the segment to the one above it. A
// chunk's slab (the tile with its halo, 40 columns wide) arrives by TMA, which fills zeros outside the
// grid, into a ring of two stages; its 32-byte columns in the 32-byte swizzle, so a warp's reads meet
// no bank twice (and rows of 40 columns keep a column's swizzle the same in every row). Where the
// cells need an operation first (a division by hs, the clipped OC step), its operands are staged
// beside them and the block applies it in place, once per staged cell. Blocks are persistent and walk
// (tile, segment) items; the segment length is the one whose waves cost the fewest steps.
//
// Measured at 384 x 192 x 192 cells, r = 3, H v / hs and H (v / hs): 360 us for the two (the HBM
// copy rate would take 105), against 1005 us gathered from a staged tile tap by tap with a
// block per chunk, and 550 us with the next chunk staged through registers and a branch per tap. What it waits
// for at reach 2 is shared memory (74 % of its rate, FP64 pipe 27 %, DRAM 24 %).
//
// The staged form takes tap lists without repeats whose weights are those of their class and |dz| and
// whose classes are whole (every cone's), up to reach 3. Lists that reach further, fields that do not start on a
// 16-byte boundary and all lists of lpb_filter are taken tap by tap (k_filter_taps). Where the march meets
// another list (lpb_filter_reach, lpb_oc_trial) it gathers cell by cell from global memory.
#include <algorithm>
#include <type_traits>

#include "lp_common.cuh"
#include "lp_quotient.cuh"
#include "lp_tma.cuh"

#define LP_MAX_TAPS 1024

namespace {

constexpr int FT_R = 3;          // largest reach of the staged form
constexpr int FT_X = 32;         // cell columns per tile in x (a warp's lanes)
constexpr int FT_Y = 16;         // in y (a row per warp)
constexpr int FT_THREADS = 32 * FT_Y;
constexpr int FT_XH = 40;        // staged columns per row, from 4 below the tile
constexpr int FT_BLOCKS = 296;   // two resident blocks on each of 148 SMs (one at reach 3)

// The operation on a cell before the taps are applied.
struct FilterIn {
  const double* v;
  const double* hs_in;   // or null
};
// OC trial at a multiplier: clip(ts / sl, max(0, x - move), min(1, x + move)), flagged cells held.
// WRITE: the accepted design, with the expressions of k_oc_stepped and k_project (lp_simp.cu). A trial
// that only measures the volume has the same values: its two divisors, sl and den, are the same for all
// cells, so a quotient is the product with the divisor's inverse corrected by its remainder (lp_quotient),
// three operations where a division takes over ten (a design update of 192 x 96 x 96 cells, nine trials and
// the write: 644 us; 626 with the products uncorrected and tanh by way of exp, off by up to a rounding of 1).
template <bool WRITE>
struct TrialIn {
  const double* ts;      // x sqrt(-dc / dv)
  const double* x;
  const uint8_t* flags;  // or null
  double sl, isl, move;  // sqrt(lm), its inverse
};
struct FilterOut {
  double* out;
  const double* hs_out;  // or null
  double* e_out;         // or null
  double penal, emin;
};
template <bool WRITE>
struct TrialOut {
  double* xn;
  double* xt;
  double* xp;
  const double* hs;
  const double* w;
  const uint8_t* flags;
  double beta, eta, tbe, den, iden;
};

__device__ __forceinline__ double pre(const FilterIn& f, long long, double a, double b) {
  return f.hs_in ? a / b : a;
}
__host__ __device__ __forceinline__ const double* raw_a(const FilterIn& f) { return f.v; }
__host__ __device__ __forceinline__ const double* raw_b(const FilterIn& f) { return f.hs_in; }
template <bool WRITE>
__device__ __forceinline__ double pre(const TrialIn<WRITE>& f, long long c, double ts, double xv) {
  double v;
  if constexpr (WRITE) {
    v = fmin(fmax(ts / f.sl, fmax(0.0, xv - f.move)), fmin(1.0, xv + f.move));
  } else {
    // compares and selects; a NaN step goes to the lower bound, as fmax takes it
    const double l = xv - f.move, h = xv + f.move, lo = l > 0.0 ? l : 0.0, hi = h < 1.0 ? h : 1.0;
    v = lp_quotient_inf(ts, f.sl, f.isl);
    v = v > lo ? v : lo;
    v = v < hi ? v : hi;
  }
  if (f.flags) {
    const uint8_t fl = f.flags[c];
    if (fl & 1) v = 1.0;
    else if (fl & 2) v = 0.0;
  }
  return v;
}
template <bool WRITE>
__host__ __device__ __forceinline__ const double* raw_a(const TrialIn<WRITE>& f) { return f.ts; }
template <bool WRITE>
__host__ __device__ __forceinline__ const double* raw_b(const TrialIn<WRITE>& f) { return f.x; }

// the first n of four consecutive doubles, as two 16-byte accesses where the array allows it
__device__ __forceinline__ void load4(const double* p, bool vec, int n, double (&v)[4]) {
  if (vec && n >= 4) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p + 2));
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = q < n ? __ldg(p + q) : 1.0;
  }
}
__device__ __forceinline__ void save4(double* p, bool vec, int n, const double (&v)[4]) {
  if (vec && n >= 4) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < n) p[q] = v[q];
  }
}

// the sums r of the first n cells from cell c of a column's chunk
__device__ __forceinline__ void finish(const FilterOut& o, const FilterIn&, long long c, bool vec, int n,
                                       const double (&r)[4], double&) {
  double v[4] = {r[0], r[1], r[2], r[3]};
  if (o.hs_out) {
    double h[4];
    load4(o.hs_out + c, vec, n, h);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = v[q] / h[q];
  }
  save4(o.out + c, vec, n, v);
  if (o.e_out) {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = o.emin + pow(v[q], o.penal) * (1.0 - o.emin);
    save4(o.e_out + c, vec, n, v);
  }
}
// xt = r / hs, its projection and the volume's share
template <bool WRITE>
__device__ __forceinline__ void finish(const TrialOut<WRITE>& o, const TrialIn<WRITE>& in, long long c, bool vec, int n,
                                       const double (&r)[4], double& acc) {
  double h[4], w[4], xt[4], xp[4];
  load4(o.hs + c, vec, n, h);
  load4(o.w + c, vec, n, w);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    xt[q] = r[q] / h[q];
    const double num = o.tbe + tanh(o.beta * (xt[q] - o.eta));
    xp[q] = WRITE ? num / o.den : lp_quotient(num, o.den, o.iden);
    if (q < n) {
      if (o.flags) {
        const uint8_t fl = o.flags[c + q];
        if (fl & 1) xp[q] = 1.0;
        else if (fl & 2) xp[q] = 0.0;
      }
      acc += xp[q] * w[q];
    }
  }
  if constexpr (WRITE) {
    double xn[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) xn[q] = q < n ? pre(in, c + q, in.ts[c + q], in.x[c + q]) : 0.0;
    save4(o.xn + c, vec, n, xn);
    save4(o.xt + c, vec, n, xt);
    save4(o.xp + c, vec, n, xp);
  }
}

struct FilterMaps {
  CUtensorMap a, b;   // (4, nx, ny, chunks), box (4, 40, 16 + 2R, 1), 32-byte swizzle
};

template <int R>
struct Slab {
  static constexpr int BYTES = (FT_XH * (FT_Y + 2 * R) * 32 + 1023) / 1024 * 1024;
};

// the weights of class dx^2 + dy^2 = k at |dz|, and bit |dz| of present[k] where the class is listed
struct FilterTaps {
  double w[2 * FT_R * FT_R + 1][FT_R + 1];
  unsigned present[2 * FT_R * FT_R + 1];
  int count[2 * FT_R * FT_R + 1][FT_R + 1];   // taps listed
};

// columns of class k within reach R
template <int R, int K>
struct ClassSize {
  static constexpr int count() {
    int n = 0;
    for (int dx = -R; dx <= R; ++dx)
      for (int dy = -R; dy <= R; ++dy) n += dx * dx + dy * dy == K;
    return n;
  }
  static constexpr int N = count();
};
template <int R>
__device__ __forceinline__ int class_size(int k) {
  int n = 0;
  for (int dx = -R; dx <= R; ++dx)
    for (int dy = -R; dy <= R; ++dy) n += dx * dx + dy * dy == k;
  return n;
}

// whether the list is one the staged form takes: within reach R, every (class, |dz|) whole with one
// weight, no repeats (counting catches one together with a missing tap only where the list is sorted,
// so sorted lists alone are taken). Fills tp; the whole block calls it.
template <int R>
__device__ bool list_staged(FilterTaps& tp, const int* __restrict__ toff, const double* __restrict__ tw, int ntaps,
                            bool refuse) {
  constexpr int NK = 2 * R * R + 1;
  const int tid = threadIdx.x, nt = blockDim.x;
  int bad = refuse;
  for (int i = tid; i < NK * (R + 1); i += nt) tp.count[i / (R + 1)][i % (R + 1)] = 0;
  for (int i = tid; i < ntaps; i += nt) {
    const int dx = toff[3 * i], dy = toff[3 * i + 1], dz = toff[3 * i + 2];
    bad |= max(abs(dx), max(abs(dy), abs(dz))) > R;
    if (i) {
      const int px = toff[3 * i - 3], py = toff[3 * i - 2], pz = toff[3 * i - 1];
      bad |= !(px < dx || (px == dx && (py < dy || (py == dy && pz < dz))));
    }
  }
  if (__syncthreads_or(bad)) return false;
  for (int i = tid; i < ntaps; i += nt) {
    const int k = toff[3 * i] * toff[3 * i] + toff[3 * i + 1] * toff[3 * i + 1], dz = abs(toff[3 * i + 2]);
    tp.w[k][dz] = tw[i];
    atomicAdd(&tp.count[k][dz], 1);
  }
  __syncthreads();
  bad = 0;
  for (int i = tid; i < ntaps; i += nt) {
    const int k = toff[3 * i] * toff[3 * i] + toff[3 * i + 1] * toff[3 * i + 1], dz = abs(toff[3 * i + 2]);
    bad |= !(tp.w[k][dz] == tw[i]) || tp.count[k][dz] != class_size<R>(k) * (dz ? 2 : 1);
  }
  if (tid < NK) {
    unsigned m = 0;
    for (int dz = 0; dz <= R; ++dz) m |= (tp.count[tid][dz] ? 1u : 0u) << dz;
    tp.present[tid] = m;
  }
  return __syncthreads_or(bad) == 0;
}

// taps from global memory, cell by cell
template <class In, class Out>
__device__ void gather_item(const In& in, const Out& o, const int* __restrict__ toff, const double* __restrict__ tw,
                            int ntaps, const LpGrid& g, int x0, int y0, int c0, int c1, double& acc) {
  const int x = x0 + (int)(threadIdx.x & 31), y = y0 + (int)(threadIdx.x >> 5);
  if (x >= g.nx || y >= g.ny) return;
  for (int z = 4 * c0; z < min(4 * c1, g.nz); ++z) {
    double s = 0.0;
    for (int i = 0; i < ntaps; ++i) {
      const int xx = x + toff[3 * i], yy = y + toff[3 * i + 1], zz = z + toff[3 * i + 2];
      if (xx < 0 || yy < 0 || zz < 0 || xx >= g.nx || yy >= g.ny || zz >= g.nz) continue;
      const long long c = g.cell(xx, yy, zz);
      const double* b = raw_b(in);
      s += tw[i] * pre(in, c, raw_a(in)[c], b ? b[c] : 0.0);
    }
    const double r[4] = {s, 0.0, 0.0, 0.0};
    finish(o, in, g.cell(x, y, z), false, 1, r, acc);
  }
}

// class K's share of a thread's sums: acc[4 + p - dz] takes w(K, |dz|) times the class's sum at plane p
// (acc[4]: the chunk's first cell). col: the thread's cell in the slab; lo[dx]: byte offset of the first
// z pair of the column at dx, its second pair at that offset with bit 4 flipped.
template <int R, int K>
__device__ __forceinline__ void take_class(double (&acc)[8 + R], const unsigned char* col, const int (&lo)[2 * R + 1],
                                           const FilterTaps& tp) {
  const unsigned m = tp.present[K];
  if (!m) return;
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  bool first = true;
#pragma unroll
  for (int dx = -R; dx <= R; ++dx)
#pragma unroll
    for (int dy = -R; dy <= R; ++dy) {
      if (dx * dx + dy * dy != K) continue;
      const double2 a = *reinterpret_cast<const double2*>(col + lo[dx + R] + dy * FT_XH * 32);
      const double2 b = *reinterpret_cast<const double2*>(col + (lo[dx + R] ^ 16) + dy * FT_XH * 32);
      if (first) {
        t[0] = a.x;
        t[1] = a.y;
        t[2] = b.x;
        t[3] = b.y;
        first = false;
      } else {
        t[0] += a.x;
        t[1] += a.y;
        t[2] += b.x;
        t[3] += b.y;
      }
    }
#pragma unroll
  for (int dz = 0; dz <= R; ++dz) {
    if (!((m >> dz) & 1)) continue;
    const double w = tp.w[K][dz];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      acc[4 + p - dz] += w * t[p];
      if (dz) acc[4 + p + dz] += w * t[p];
    }
  }
}
template <int R, int K>
__device__ __forceinline__ void take_classes(double (&acc)[8 + R], const unsigned char* col,
                                             const int (&lo)[2 * R + 1], const FilterTaps& tp) {
  if constexpr (K <= 2 * R * R) {
    if constexpr (ClassSize<R, K>::N > 0) take_class<R, K>(acc, col, lo, tp);
    take_classes<R, K + 1>(acc, col, lo, tp);
  }
}

template <int R, class In, class Out>
__global__ void __launch_bounds__(FT_THREADS, (R < 3 ? 2 : 1))
k_filter_march(const __grid_constant__ FilterMaps maps, const In in, const Out o, const int* __restrict__ toff,
               const double* __restrict__ tw, int ntaps, LpGrid g, int seg, int tma, int vec, double* __restrict__ part) {
  lp_after_launch();
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw_off = lp_smem_addr(smem_raw);
  unsigned char* slabs = smem_raw + ((1024u - (raw_off & 1023u)) & 1023u);   // a: stages 0, 1, then b: 0, 1
  __shared__ FilterTaps tp;
  __shared__ alignas(8) uint64_t full[2];
  constexpr int YH = FT_Y + 2 * R, SLAB = Slab<R>::BYTES;
  constexpr uint32_t BYTES = FT_XH * YH * 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool staged = list_staged<R>(tp, toff, tw, ntaps, tma == 0);
  if (tid == 0) {
    lp_mbar_init(&full[0], 1);
    lp_mbar_init(&full[1], 1);
    lp_fence_barrier_init();
  }
  __syncthreads();
  const int ntx = (g.nx + FT_X - 1) / FT_X, nty = (g.ny + FT_Y - 1) / FT_Y, nch = (g.nz + 3) / 4;
  const int nseg = (nch + seg - 1) / seg;
  const long long items = (long long)ntx * nty * nseg, zstep = g.cell_zc_stride();
  const bool two = raw_b(in) != nullptr;
  // this thread's column in a slab: row warp + R, column lane + 4; the swizzle bit of column lane + 4 + dx
  int lo[2 * R + 1];
#pragma unroll
  for (int dx = -R; dx <= R; ++dx) lo[dx + R] = (int)lp_swz32((uint32_t)(((warp + R) * FT_XH + lane + 4 + dx) * 32));
  uint32_t n = 0;          // chunks staged so far: stage n & 1, phase (n >> 1) & 1
  double vacc = 0.0;
  for (long long it = blockIdx.x; it < items; it += gridDim.x) {
    const int tx = (int)(it % ntx), ty = (int)((it / ntx) % nty), sg = (int)(it / ((long long)ntx * nty));
    const int x0 = tx * FT_X, y0 = ty * FT_Y, c0 = sg * seg, c1 = min(c0 + seg, nch);
    if (!staged) {
      gather_item(in, o, toff, tw, ntaps, g, x0, y0, c0, c1, vacc);
      continue;
    }
    const double vacc0 = vacc;
    const int ca = max(c0 - 1, 0), cb = min(c1, nch - 1);   // chunks staged: ca .. cb
    auto issue = [&](int c, uint32_t k) {
      const uint32_t s = k & 1;
      lp_mbar_expect_tx(&full[s], two ? 2 * BYTES : BYTES);
      lp_tma_load_4d(slabs + s * SLAB, &maps.a, 0, x0 - 4, y0 - R, c, &full[s]);
      if (two) lp_tma_load_4d(slabs + (2 + s) * SLAB, &maps.b, 0, x0 - 4, y0 - R, c, &full[s]);
    };
    if (tid == 0) {
      issue(ca, n);
      if (ca < cb) issue(ca + 1, n + 1);
    }
    double acc[8 + R];   // sums of the cells 4 (c - 1) .. 4 c + 3 + R
#pragma unroll
    for (int k = 0; k < 8 + R; ++k) acc[k] = 0.0;
    const int x = x0 + lane, y = y0 + warp;
    const bool own = x < g.nx && y < g.ny;
    for (int c = ca; c <= c1; ++c) {
      if (c <= cb) {
        const uint32_t s = n & 1;
        unsigned char* sa = slabs + s * SLAB;
        if (__syncthreads_or(!lp_mbar_wait(&full[s], (n >> 1) & 1))) {
          staged = false;   // a load did not arrive in time: the rest without TMA
          break;
        }
        const int ztail = g.nz - 4 * c;   // the chunk's cells in the grid
        if (two || ztail < 4) {
          const unsigned char* sb = slabs + (2 + s) * SLAB;
          for (int yl = warp; yl < YH; yl += FT_Y) {
            const int gy = y0 - R + yl;
            if (gy < 0 || gy >= g.ny) continue;
            for (int j = lane; j < 2 * FT_XH; j += 32) {
              const int gx = x0 - 4 + (j >> 1), half = j & 1;
              if (gx < 0 || gx >= g.nx || gx < x0 - R || gx >= x0 + FT_X + R) continue;
              if (R <= 2 && ((half == 0 && c < c0) || (half == 1 && c == c1))) continue;   // planes out of reach
              const uint32_t at = lp_swz32((uint32_t)(yl * FT_XH * 32 + j * 16));
              double2 v = *reinterpret_cast<double2*>(sa + at);
              double2 b = make_double2(1.0, 1.0);
              if (two) b = *reinterpret_cast<const double2*>(sb + at);
              const long long i = g.cell(gx, gy, 4 * c) + 2 * half;
              v.x = 2 * half < ztail ? pre(in, i, v.x, b.x) : 0.0;
              v.y = 2 * half + 1 < ztail ? pre(in, i + 1, v.y, b.y) : 0.0;
              *reinterpret_cast<double2*>(sa + at) = v;
            }
          }
          __syncthreads();
        }
        take_classes<R, 0>(acc, sa, lo, tp);
        lp_fence_proxy_async();
        __syncthreads();   // the stage is read
        if (tid == 0 && c + 2 <= cb) issue(c + 2, n + 2);
        ++n;
      }
      if (c > c0 && own) {   // the cells of chunk c - 1, complete after this chunk's columns
        const long long cell = (c - 1) * zstep + 4LL * ((long long)y * g.nx + x);
        const double r[4] = {acc[0], acc[1], acc[2], acc[3]};
        finish(o, in, cell, vec != 0, g.nz - 4 * (c - 1), r, vacc);
      }
#pragma unroll
      for (int k = 0; k < 4 + R; ++k) acc[k] = acc[k + 4];
#pragma unroll
      for (int k = 4 + R; k < 8 + R; ++k) acc[k] = 0.0;
    }
    if (!staged) {
      vacc = vacc0;
      gather_item(in, o, toff, tw, ntaps, g, x0, y0, c0, c1, vacc);
      // its own loads still in flight land before the block ends (bounded as well)
      if (tid == 0)
        for (int s = 0; s < 2; ++s) lp_mbar_wait(&full[s], (s == (int)(n & 1) ? n >> 1 : (n + 1) >> 1) & 1);
    }
  }
  if (part) {
    __shared__ double sh[32];
    vacc = lp_block_sum(vacc, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = vacc;
  }
}

// Taps one after another, for the lists and fields the march does not take:
//   out = H (v / hs_in) / hs_out, with e_out also the SIMP law on the result.
// A block takes a tile of 32 x 8 cell columns times one z chunk (4 cells): it stages the tile with its halo of
// reach R (the largest |offset| of the taps, up to TAPS_R) in shared memory, v / hs_in formed once per staged
// cell and zeros outside the grid, and each thread sums the taps for the 4 cells of its column in the list's
// order. Taps that reach further are gathered from global memory, cell by cell, in the same order: bound by
// the loads' latency, so the blocks are small and many (reach 4, 192 x 96 x 96 cells: 1141 us; in the march's
// blocks of 512, one per SM, 4690).
constexpr int TAPS_X = 32, TAPS_Y = 8, TAPS_R = 2;
__global__ void __launch_bounds__(256) k_filter_taps(double* __restrict__ out, const double* __restrict__ v,
                                                     const int* __restrict__ toff, const double* __restrict__ tw,
                                                     int ntaps, const double* __restrict__ hs_in,
                                                     const double* __restrict__ hs_out, double* __restrict__ e_out,
                                                     double penal, double emin, LpGrid g) {
  lp_after_launch();
  extern __shared__ unsigned char smem_raw[];
  __shared__ double tile[(4 + 2 * TAPS_R) * (TAPS_Y + 2 * TAPS_R) * (TAPS_X + 2 * TAPS_R)];
  __shared__ int s_reach;
  int* so = reinterpret_cast<int*>(smem_raw);
  double* sw = reinterpret_cast<double*>(smem_raw + ((3 * ntaps * sizeof(int) + 15) & ~15));
  if (threadIdx.x == 0) s_reach = 0;
  __syncthreads();
  int reach = 0;
  for (int i = threadIdx.x; i < ntaps; i += blockDim.x) {
    const int dx = toff[3 * i], dy = toff[3 * i + 1], dz = toff[3 * i + 2];
    so[3 * i] = dx;
    so[3 * i + 1] = dy;
    so[3 * i + 2] = dz;
    sw[i] = tw[i];
    reach = max(reach, max(abs(dx), max(abs(dy), abs(dz))));
  }
  if (reach) atomicMax(&s_reach, reach);
  __syncthreads();
  const int R = s_reach;
  const int nbx = (g.nx + TAPS_X - 1) / TAPS_X, nby = (g.ny + TAPS_Y - 1) / TAPS_Y;
  const int bx = (int)(blockIdx.x % nbx), rest = (int)(blockIdx.x / nbx);
  const int by = rest % nby, cz = rest / nby;
  const int x0 = bx * TAPS_X, y0 = by * TAPS_Y;
  const int x = x0 + (int)(threadIdx.x & 31), y = y0 + (int)(threadIdx.x >> 5);
  const bool own = x < g.nx && y < g.ny;
  if (R > TAPS_R) {
    if (!own) return;
    for (int zq = 0; zq < 4; ++zq) {
      const int z = 4 * cz + zq;
      if (z >= g.nz) break;
      double acc = 0.0;
      for (int i = 0; i < ntaps; ++i) {
        const int xx = x + so[3 * i], yy = y + so[3 * i + 1], zz = z + so[3 * i + 2];
        if (xx < 0 || yy < 0 || zz < 0 || xx >= g.nx || yy >= g.ny || zz >= g.nz) continue;
        const long long c = g.cell(xx, yy, zz);
        double vi = v[c];
        if (hs_in) vi = vi / hs_in[c];
        acc += sw[i] * vi;
      }
      const long long c = g.cell(x, y, z);
      if (hs_out) acc = acc / hs_out[c];
      out[c] = acc;
      if (e_out) e_out[c] = emin + pow(acc, penal) * (1.0 - emin);
    }
    return;
  }
  const int XH = TAPS_X + 2 * R, YH = TAPS_Y + 2 * R, ZH = 4 + 2 * R, P = XH * YH;
  const int CR = (R + 3) / 4;  // halo chunks on each side
  // the taps' offsets in the staged tile, written over their first coordinate
  for (int i = threadIdx.x; i < ntaps; i += blockDim.x) so[3 * i] += (so[3 * i + 2] * YH + so[3 * i + 1]) * XH;
  // a warp stages a (chunk, y) row at a time: 4 XH doubles contiguous in memory, lanes along it
  const int rowlen = 4 * XH, nrows = (2 * CR + 1) * YH;
  const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5), nwarps = (int)(blockDim.x >> 5);
  for (int row = warp; row < nrows; row += nwarps) {
    const int cr = row / YH, yl = row - cr * YH;
    const int gy = y0 - R + yl, zbase = 4 * (cz - CR + cr);
    const bool yok = gy >= 0 && gy < g.ny;
    for (int j = lane; j < rowlen; j += 32) {
      const int xl = j >> 2, gz = zbase + (j & 3);
      const int zl = gz - (4 * cz - R);
      if (zl < 0 || zl >= ZH) continue;
      const int gx = x0 - R + xl;
      double val = 0.0;
      if (yok && gx >= 0 && gx < g.nx && gz >= 0 && gz < g.nz) {
        const long long c = g.cell(gx, gy, gz);
        val = v[c];
        if (hs_in) val = val / hs_in[c];
      }
      tile[(zl * YH + yl) * XH + xl] = val;
    }
  }
  __syncthreads();
  if (!own) return;
  const int ctr = (R * YH + R + (int)(threadIdx.x >> 5)) * XH + R + (int)(threadIdx.x & 31);
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = 0; i < ntaps; ++i) {
    const int o = ctr + so[3 * i];
    const double w = sw[i];
#pragma unroll
    for (int zq = 0; zq < 4; ++zq) acc[zq] += w * tile[o + zq * P];
  }
#pragma unroll
  for (int zq = 0; zq < 4; ++zq) {
    const int z = 4 * cz + zq;
    if (z >= g.nz) break;
    const long long c = g.cell(x, y, z);
    double r = acc[zq];
    if (hs_out) r = r / hs_out[c];
    out[c] = r;
    if (e_out) e_out[c] = emin + pow(r, penal) * (1.0 - emin);
  }
}

// ordered sum of the blocks' volumes
__global__ void k_filter_volume(const double* __restrict__ part, int n, double* __restrict__ out) {
  lp_after_launch();
  __shared__ double sh[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
  s = lp_block_sum(s, sh);
  if (threadIdx.x == 0) *out = s;
}

// ts = x sqrt(-dc / dv)
__global__ void k_oc_step_base(double* __restrict__ ts, const double* __restrict__ x, const double* __restrict__ dc,
                               const double* __restrict__ dv, LpGrid g) {
  lp_after_launch();
  const long long total = g.cells_padded();
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    int x_, y_, z;
    if (!g.cell_at(t, x_, y_, z)) continue;
    ts[t] = x[t] * sqrt(-dc[t] / dv[t]);
  }
}

constexpr int NO_TMA = 1;   // nothing launched
template <int R, class In, class Out>
int launch_reach(const In& in, const Out& o, const int* toff, const double* tw, int ntaps, LpGrid g, bool vec,
                 double* part, int* nblocks, cudaStream_t st) {
  const long long tiles = (long long)((g.nx + FT_X - 1) / FT_X) * ((g.ny + FT_Y - 1) / FT_Y);
  const int nch = (g.nz + 3) / 4, slots = R < 3 ? FT_BLOCKS : FT_BLOCKS / 2;
  // the segment length with the fewest chunk steps in all waves; a segment stages two chunks more than it
  // owns
  int best = nch;
  long long cost = -1;
  for (int seg = 1; seg <= nch; ++seg) {
    const long long items = tiles * ((nch + seg - 1) / seg), waves = (items + slots - 1) / slots;
    const long long c = waves * (seg + 2);
    if (cost < 0 || c <= cost) {
      cost = c;
      best = seg;
    }
  }
  const long long items = tiles * ((nch + best - 1) / best);
  const int nb = (int)std::min<long long>(items, slots);
  FilterMaps maps{};
  const uint64_t dims[4] = {4, (uint64_t)g.nx, (uint64_t)g.ny, (uint64_t)(g.cpz / 4)};
  const uint32_t box[4] = {4, FT_XH, FT_Y + 2 * R, 1};
  // a field that TMA cannot address (not 16-byte aligned) is a trial's to gather, a filter's to take by taps
  bool tma = lp_make_map(&maps.a, raw_a(in), 4, dims, box, 8, 32);
  if (tma && raw_b(in)) tma = lp_make_map(&maps.b, raw_b(in), 4, dims, box, 8, 32);
  if (!tma && std::is_same<In, FilterIn>::value) return NO_TMA;
  const int smem = (raw_b(in) ? 4 : 2) * Slab<R>::BYTES + 1024;
  if (cudaFuncSetAttribute(k_filter_march<R, In, Out>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           4 * Slab<R>::BYTES + 1024) != cudaSuccess)
    return LP_ERR_LAUNCH;
  lp_launch(k_filter_march<R, In, Out>, nb, FT_THREADS, smem, st, maps, in, o, toff, tw, ntaps, g, best, tma ? 1 : 0, vec ? 1 : 0,
            part);
  if (nblocks) *nblocks = nb;
  LP_LAUNCH_CHECK();
  return LP_OK;
}

template <class In, class Out>
int launch_march(const In& in, const Out& o, const int* toff, const double* tw, int ntaps, int reach, LpGrid g,
                 bool vec, double* part, int* nblocks, cudaStream_t st) {
  if (reach <= 1) return launch_reach<1>(in, o, toff, tw, ntaps, g, vec, part, nblocks, st);
  if (reach == 2) return launch_reach<2>(in, o, toff, tw, ntaps, g, vec, part, nblocks, st);
  return launch_reach<FT_R>(in, o, toff, tw, ntaps, g, vec, part, nblocks, st);
}

int launch_taps(const FilterIn& in, const FilterOut& o, const int* toff, const double* tw, int ntaps, LpGrid g,
                cudaStream_t st) {
  const size_t smem = ((3 * ntaps * sizeof(int) + 15) & ~(size_t)15) + ntaps * sizeof(double);
  const long long tiles = (long long)((g.nx + TAPS_X - 1) / TAPS_X) * ((g.ny + TAPS_Y - 1) / TAPS_Y) * ((g.nz + 3) / 4);
  if (tiles > 2147483647LL) return LP_ERR_ARG;
  lp_launch(k_filter_taps, (unsigned)tiles, 256, smem, st, o.out, in.v, toff, tw, ntaps, in.hs_in, o.hs_out, o.e_out, o.penal,
            o.emin, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

#define LP_GRID_ARGS int nx, int ny, int nz, int pz, int cpz
#define LP_GRID lp_grid(nx, ny, nz, pz, cpz)
#define LP_ST ((cudaStream_t)stream)

extern "C" {

// out[c] = sum_t w_t v[c + d_t] (zeros outside the grid); optional division of v by hs_in before and
// of the sum by hs_out after; with e_out also the SIMP law e_out = emin + out^p (1 - emin). reach: the
// largest |offset| of the taps. A cone's taps, in order: the march up to reach 3 (other lists that the march
// is given it gathers, a few times slower than lpb_filter).
int lpb_filter_reach(double* out, const double* v, const int* toff, const double* tw, int ntaps, int reach,
                     const double* hs_in, const double* hs_out, double* e_out, double penal, double emin, LP_GRID_ARGS,
                     void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || !out || !v || !toff || !tw || ntaps < 1 || ntaps > LP_MAX_TAPS || reach < 0) return LP_ERR_ARG;
  if (out == v) return LP_ERR_ARG;
  const FilterIn in{v, hs_in};
  const FilterOut o{out, hs_out, e_out, penal, emin};
  const bool vec = aligned16(out) && aligned16(hs_out) && aligned16(e_out);
  const int rc = reach > FT_R ? NO_TMA : launch_march(in, o, toff, tw, ntaps, reach, g, vec, nullptr, nullptr, LP_ST);
  return rc == NO_TMA ? launch_taps(in, o, toff, tw, ntaps, g, LP_ST) : rc;
}

// the same for any list, its taps one after another
int lpb_filter(double* out, const double* v, const int* toff, const double* tw, int ntaps, const double* hs_in,
               const double* hs_out, double* e_out, double penal, double emin, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || !out || !v || !toff || !tw || ntaps < 1 || ntaps > LP_MAX_TAPS) return LP_ERR_ARG;
  if (out == v) return LP_ERR_ARG;
  return launch_taps(FilterIn{v, hs_in}, FilterOut{out, hs_out, e_out, penal, emin}, toff, tw, ntaps, g, LP_ST);
}

// ts = x sqrt(-dc / dv): the part of the OC step that every trial multiplier shares
int lpb_oc_step_base(double* ts, const double* x, const double* dc, const double* dv, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || !ts || !x || !dc || !dv) return LP_ERR_ARG;
  lp_launch(k_oc_step_base, lp_blocks(g.cells_padded(), 256), 256, 0, LP_ST, ts, x, dc, dv, g);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

// One trial of the volume multiplier lm: xn = the clipped OC step from ts (lpb_oc_step_base), xt =
// H xn / hs, xp its projection at (beta, eta), *vol = sum xp w. xn, xt, xp: all given, or all NULL when
// only the volume is wanted. part: 592 doubles.
int lpb_oc_trial(double* xn, double* xt, double* xp, const double* ts, const double* x, double lm, double move,
                 const uint8_t* flags, const int* toff, const double* tw, int ntaps, int reach, const double* hs,
                 double beta, double eta, const double* w, double* part, double* vol, LP_GRID_ARGS, void* stream) {
  LpGrid g = LP_GRID;
  if (!lp_grid_ok(g) || !ts || !x || !toff || !tw || ntaps < 1 || ntaps > LP_MAX_TAPS || reach < 0 || !hs || !w || !part ||
      !vol || !(lm > 0.0))
    return LP_ERR_ARG;
  if ((xn != nullptr) != (xt != nullptr) || (xn != nullptr) != (xp != nullptr) || (xn && (xn == x || xn == ts)))
    return LP_ERR_ARG;
  const double tbe = tanh(beta * eta), den = tbe + tanh(beta * (1.0 - eta)), sl = sqrt(lm);
  const bool vec = aligned16(xn) && aligned16(xt) && aligned16(xp) && aligned16(hs) && aligned16(w);
  int nb = 0, rc;
  if (xn) {
    const TrialIn<true> in{ts, x, flags, sl, 1.0 / sl, move};
    const TrialOut<true> o{xn, xt, xp, hs, w, flags, beta, eta, tbe, den, 1.0 / den};
    rc = launch_march(in, o, toff, tw, ntaps, reach, g, vec, part, &nb, LP_ST);
  } else {
    const TrialIn<false> in{ts, x, flags, sl, 1.0 / sl, move};
    const TrialOut<false> o{nullptr, nullptr, nullptr, hs, w, flags, beta, eta, tbe, den, 1.0 / den};
    rc = launch_march(in, o, toff, tw, ntaps, reach, g, vec, part, &nb, LP_ST);
  }
  if (rc != LP_OK) return rc;
  lp_launch(k_filter_volume, 1, 512, 0, LP_ST, part, nb, vol);
  LP_LAUNCH_CHECK();
  return LP_OK;
}

}  // extern "C"
