// FP64 residual products of the butterfly Legendre step on the FP64 units
// (matrices of tree depth 0 and 1, see plan.h, build_fast_path).
//
// For one row group (residual blocks sharing rows [rs, rs + R) of a matrix):
//   alm2map   X[c][v] = sum_r P[r][c] a[r][v]
//   map2alm   a[r][v] = sum_c P[r][c] X[c][v]
// P[r][c] follows the three-term recurrence of column c
// (src/legendre_transform.c.in:680-716), here with a scale per row:
//   P_r = s_r y_r,   y_r = (x^2 A_r + B_r) y_{r-1} - y_{r-2},
// s_r = -gamma_r s_{r-2}, A_r = beta_r s_{r-1} / s_r, B_r = alpha_r A_r
// (program.cpp, direct_tables), so that one row of one column costs two
// fused multiply-adds and no P is ever stored: both kernels keep the
// recurrence in the registers of the thread that multiplies with it.  s_r is
// folded into the alm row (alm2map) or the finished sum (map2alm).
//
// What bounds them: the FP64 pipe.  An element costs 2 operations for the
// recurrence and one per vector, 148 SMs x 64 lanes x 1.9 GHz = 18 T/s; the
// FP64 tensor instruction (mma.m8n8k4) runs on the same units at the same
// rate (36.9 TFLOP/s measured, multiply-adds 33).  The kernels these replace
// built P tiles in shared memory with a column per thread, the row's
// coefficients read from global memory inside the dependent chain.
// Measured, nside 512, lmax 1024 (before -> now):
//               1 map               16 maps             32 maps
//   alm2map     2014 ->  194 us     4503 -> 1369 us     5735 -> 2736 us
//   map2alm     2491 ->  414 us     5387 -> 1494 us     8586 -> 2903 us
// The FP64 pipe is busy 62% of the alm2map kernel's time (broadcast reads
// keep a register-blocked loop at 76% of it at best), 57% of map2alm's.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "plan.h"

namespace wm {

namespace {

constexpr int kDirectThr = 128;  // 4 warps
constexpr int kDirectWarps = kDirectThr / 32;

__device__ __forceinline__ int64_t alm_row0(const DevMatrix &M, int lmax) {
  return (int64_t)M.m * (2 * lmax - M.m + 3) / 2 + M.odd;
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Asynchronous copies into shared memory; zeros where `in` is false.
__device__ __forceinline__ void copy16(void *dst, const void *src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy8(void *dst, const void *src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}

// ------------------------------------------------------------------------
// alm2map.  A thread owns C columns (32 apart) and NV vectors of each.  The
// CTA stages chunks of kChunk rows of the alm and of the coefficients in
// shared memory by asynchronous copies, one chunk ahead, multiplies the alm
// rows by s_r there, and every thread reads them as broadcasts: NV / 2 + 1
// 16-byte reads for C (NV + 2) multiply-adds, which is why C = 2 -- with
// C = 1 the reads, not the FP64 pipe, set the time.  Columns are sorted by
// first row: a warp enters a chunk at the first row of its own columns, and
// puts the stored first values in until its last column has started.  The
// sum over rows runs in row order for every number of vectors.
// Chunks of 32 rows took 1547 us where 128 take 1369 (16 maps, nside 512:
// the barriers around a chunk), C = 4 for 1 map 244 us against 215, and
// the tensor instruction with P in its A fragments 1430 us for 16 maps and
// 553 us for 1, whose two vectors it pads to eight.
// ------------------------------------------------------------------------
constexpr int kChunk = 128;

// CTAs per SM that the accumulators leave room for
constexpr int direct_ctas(int accumulators) {
  return accumulators > 16 ? 3 : accumulators > 8 ? 4 : accumulators > 4 ? 5 : 6;
}

template <int NV>
struct A2mChunk {
  double a[kChunk][NV];
  double2 ab[kChunk];
  double scale[kChunk];
};

template <int NV, int C>
__global__ void __launch_bounds__(kDirectThr, direct_ctas(NV * C)) k_direct_a2m(DirectParams p, int npass) {
  __shared__ __align__(16) A2mChunk<NV> s_chunk[2];
  const int tid = threadIdx.x, lane = tid & 31;
  for (int unit = blockIdx.x; unit < p.ntiles_a * npass; unit += gridDim.x) {
    const DevDirectTileA T = p.tiles_a[unit / npass];
    // a tile's first columns have the most rows: give them to another
    // scheduler's warp from tile to tile
    const int warp = ((tid >> 5) + unit) % kDirectWarps;
    const int v0 = (unit % npass) * NV, vn = min(NV, p.nvecs - v0);
    const DevGroup G = p.groups[T.group];
    const DevMatrix M = p.mats[G.matrix];
    const double *alm = p.alm_in + (alm_row0(M, p.lmax) + 2 * (int64_t)G.rs) * p.nvecs + v0;
    const int R = G.nrows;
    const DevDirectCol *cols = p.cols + G.cols + T.col0;
    const double *inj = p.inj + kDirectInj * (G.cols + T.col0);
    // rows beyond the group are not read, vectors beyond the last arrive as zeros
    auto fetch = [&](int r0, A2mChunk<NV> &to) {
      const int n = min(kChunk, R - r0);
      for (int e = tid; e < n * (NV / 2); e += kDirectThr) {
        const int k = e / (NV / 2), v = 2 * (e % (NV / 2));
        const bool in = v < vn;
        const double *src = in ? alm + 2 * (int64_t)(r0 + k) * p.nvecs + v : alm;
        if (p.aligned) {
          copy16(&to.a[k][v], src, in);
        } else {
          copy8(&to.a[k][v], src, in);
          copy8(&to.a[k][v + 1], src + 1, in);
        }
      }
      if (tid < n) {
        copy16(&to.ab[tid], p.ab + G.coef + r0 + tid, true);
        copy8(&to.scale[tid], p.scale + G.coef + r0 + tid, true);
      }
    };
    // columns of this thread
    double x2[C], y0[C], y1[C], acc[C][NV];
    int row[C];
    int w0 = INT_MAX, wf = 0;  // the warp's columns start, and dense ones end, in rows [w0, wf)
    bool dense = false;
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const int c = (warp * C + j) * 32 + lane;
      DevDirectCol col{0.0, INT_MAX, -1};
      if (c < T.ncols) col = cols[c];
      x2[j] = col.x2;
      row[j] = col.row;
      y0[j] = y1[j] = 0.0;
      if (col.start < R) {
        w0 = min(w0, col.start);
        wf = max(wf, col.start + ((col.row & kDirectDense) ? kDirectInj : 2));
        dense = dense || (col.row & kDirectDense);
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[j][v] = 0.0;
    }
    grid_wait();  // the alm, and the readers of q
    if (T.kstart < R) fetch(T.kstart, s_chunk[0]);
    w0 = __reduce_min_sync(0xffffffffu, w0);
    wf = __reduce_max_sync(0xffffffffu, wf);
    dense = __any_sync(0xffffffffu, dense);
    int b = 0;
    for (int r0 = T.kstart; r0 < R; r0 += kChunk, b ^= 1) {
      A2mChunk<NV> &now = s_chunk[b];
      const int end = min(kChunk, R - r0);
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();  // the chunk has arrived; everyone has left the other buffer
      if (r0 + kChunk < R) fetch(r0 + kChunk, s_chunk[b ^ 1]);
      for (int e = tid; e < end * (NV / 2); e += kDirectThr) {
        double2 *at = reinterpret_cast<double2 *>(&now.a[0][0]) + e;
        const double sc = now.scale[e / (NV / 2)];
        const double2 t = *at;
        *at = make_double2(t.x * sc, t.y * sc);
      }
      __syncthreads();
      // one row: y by the recurrence, `first` puts stored values in, then the products
      auto sum_row = [&](int i, auto first) {
        const double2 ab = now.ab[i];
        double a[NV];
#pragma unroll
        for (int v = 0; v < NV; v += 2) {
          const double2 t = *reinterpret_cast<const double2 *>(&now.a[i][v]);
          a[v] = t.x;
          a[v + 1] = t.y;
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const double y = first(i, j, fma(fma(x2[j], ab.x, ab.y), y1[j], -y0[j]));
          y0[j] = y1[j];
          y1[j] = y;
#pragma unroll
          for (int v = 0; v < NV; ++v) acc[j][v] = fma(y, a[v], acc[j][v]);
        }
      };
      int i = max(0, min(w0 - r0, end));
      const int mid = min(wf - r0, end);
      if (i < mid) {
        int start[C];
        double2 f[C];
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const int c = min((warp * C + j) * 32 + lane, T.ncols - 1);
          start[j] = row[j] < 0 ? INT_MAX : cols[c].start - r0;
          f[j] = *reinterpret_cast<const double2 *>(inj + kDirectInj * (int64_t)c);
        }
        if (!dense) {
#pragma unroll 2
          for (; i < mid; ++i)
            sum_row(i, [&](int i, int j, double y) {
              return i == start[j] ? f[j].x : i == start[j] + 1 ? f[j].y : y;
            });
        } else {
#pragma unroll 1
          for (; i < mid; ++i)
            sum_row(i, [&](int i, int j, double y) {
              const int k = i - start[j];
              if (k > 1 && (row[j] & kDirectDense))
                y = inj[kDirectInj * (int64_t)((warp * C + j) * 32 + lane) + min(k, kDirectInj - 1)];
              return k == 0 ? f[j].x : k == 1 ? f[j].y : y;
            });
        }
      }
#pragma unroll 4
      for (; i < end; ++i) sum_row(i, [](int, int, double y) { return y; });
    }
    double *base = G.in_q ? p.q + (int64_t)(2 * M.m + M.odd) * p.q_mstride : p.xbuf + M.xrow * p.nvecs;
    const int64_t rstride = G.in_q ? p.q_rstride : p.nvecs;
#pragma unroll
    for (int j = 0; j < C; ++j) {
      if ((warp * C + j) * 32 + lane >= T.ncols) continue;
      double *dst = base + (int64_t)(row[j] & ~kDirectDense) * rstride + v0;
      if (p.aligned) {
#pragma unroll
        for (int v = 0; v < NV; v += 2)
          if (v < vn) *reinterpret_cast<double2 *>(dst + v) = make_double2(acc[j][v], acc[j][v + 1]);
      } else {
#pragma unroll
        for (int v = 0; v < NV; ++v)
          if (v < vn) dst[v] = acc[j][v];
      }
    }
    __syncthreads();  // the buffers are free for the next unit
  }
}

// ------------------------------------------------------------------------
// map2alm.  A unit is one row tile of a group, 8 segments of S <= kDirectSeg
// rows.  In step i the warp multiplies the 8 rows {segment g, row i} x 4
// columns by 4 columns x 8 vectors with one mma.m8n8k4 per 8 vectors; lane
// 4 g + t supplies P at (segment g, row i) of column t, so it runs the
// recurrence of its own (segment, column) from the stored seeds (y at the
// segment's first two rows) step by step, and P goes from the recurrence's
// register into the multiplication.  Steps run in blocks of four (S is a
// multiple of four), whose coefficients are read ahead of the block.  The
// four warps take every fourth group of 4 columns and add their sums in a
// fixed order, the same for every number of vectors.
//
// Columns are sorted by first row, so those that have started by the tile's
// first row are a prefix: its groups of four run a loop without any check,
// the next group's seeds and X rows and the one after's column data in
// flight.  The others put their stored first values in as the rows come.
// Segments of 8 rows (less padding, twice the column visits) took 2101 us
// where 16 take 1494 (16 maps, nside 512); copying seeds and X rows ahead
// through shared memory 1898 us.
// ------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(kDirectThr, NT == 2 ? 3 : 4) k_direct_m2a(DirectParams p, int npass) {
  constexpr int NV = 8 * NT;
  __shared__ __align__(16) double2 s_ab[kDirectSeg * 8];
  __shared__ __align__(16) double s_red[kDirectWarps][kDirectSeg * 8][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  for (int unit = blockIdx.x; unit < p.ntiles_b * npass; unit += gridDim.x) {
    const DevDirectTileB T = p.tiles_b[unit / npass];
    const int v0 = (unit % npass) * NV, vn = min(NV, p.nvecs - v0);
    const DevGroup G = p.groups[T.group];
    const DevMatrix M = p.mats[G.matrix];
    const int S = T.seg, R = G.nrows;
    const double *Xb = (G.in_q ? p.q_in + (int64_t)(2 * M.m + M.odd) * p.q_mstride : p.xbuf + M.xrow * p.nvecs) + v0;
    const int64_t rstride = G.in_q ? p.q_rstride : p.nvecs;
    // coefficients, row i of segment g at [8 i + g]
    for (int e = tid; e < 8 * S; e += kDirectThr) {
      const int r = T.row0 + (e & 7) * S + (e >> 3);
      s_ab[e] = r < R ? p.ab[G.coef + r] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    grid_wait();  // q~ or X, and the readers of the alm
    const DevDirectCol *cols = p.cols + G.cols;
    const double2 *seeds = p.seeds + T.seeds + lane;
    const int ncg = (T.nact + 3) >> 2, nfull = T.nfull >> 2, r0 = T.row0 + g * S;
    // vector of this lane's X entries; sums of vectors beyond the last are not stored
    int xv[NT];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xv[nt] = min(8 * nt + g, vn - 1);
    double acc[kDirectSeg][NT][2];
#pragma unroll
    for (int i = 0; i < kDirectSeg; ++i)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) acc[i][nt][0] = acc[i][nt][1] = 0.0;
    // The tile's rows of one group of columns; first(step, y) puts stored values in.
    auto multiply = [&](double x2, double2 seed, const double (&x)[NT], auto first) {
      double y0 = seed.x, y1 = seed.y;
      double2 ab[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) ab[i] = s_ab[8 * i + g];
#pragma unroll
      for (int k = 0; k < kDirectSeg / 4; ++k) {
        if (4 * k >= S) break;
        double y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (k == 0 && i == 0) {
            y[i] = y0 = first(0, y0);
          } else if (k == 0 && i == 1) {
            y[i] = y1 = first(1, y1);
          } else {
            y[i] = first(4 * k + i, fma(fma(x2, ab[i].x, ab[i].y), y1, -y0));
            y0 = y1;
            y1 = y[i];
          }
        }
        if (k + 1 < kDirectSeg / 4) {
#pragma unroll
          for (int i = 0; i < 4; ++i) ab[i] = s_ab[8 * (4 * (k + 1) + i) + g];  // unused past the last block
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) dmma(acc[4 * k + i][nt], y[i], x[nt]);
      }
    };
    auto load_x = [&](const DevDirectCol &c, double (&x)[NT]) {
      const double *src = Xb + (int64_t)(c.row & ~kDirectDense) * rstride;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) x[nt] = src[xv[nt]];
    };
    // groups of columns that have all started
    if (warp < nfull) {
      const DevDirectCol *pc = cols + 4 * warp + t;
      const double2 *ps = seeds + 32 * warp;
      DevDirectCol col = *pc, next = col;
      if (warp + kDirectWarps < nfull) next = pc[4 * kDirectWarps];
      double x[NT];
      load_x(col, x);
      double2 seed = *ps;
      for (int cg = warp; cg < nfull; cg += kDirectWarps) {
        pc += 4 * kDirectWarps;
        ps += 32 * kDirectWarps;
        DevDirectCol after = next;
        double xn[NT];
        double2 seedn = seed;
        load_x(next, xn);
        if (cg + kDirectWarps < nfull) seedn = *ps;
        if (cg + 2 * kDirectWarps < nfull) after = pc[4 * kDirectWarps];
        multiply(col.x2, seed, x, [](int, double y) { return y; });
        col = next;
        next = after;
        seed = seedn;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) x[nt] = xn[nt];
      }
    }
    // the others: columns that start inside the tile, or dense ones (columns
    // beyond nact have zero seeds and repeat the last one's data)
    const int other = nfull + ((warp - nfull) & (kDirectWarps - 1));
    if (other < ncg) {
      auto column = [&](int cg) { return min(4 * cg + t, T.nact - 1); };
      auto load_first = [&](int cg) {
        return *reinterpret_cast<const double2 *>(p.inj + kDirectInj * (G.cols + column(cg)));
      };
      DevDirectCol col = cols[column(other)], next = cols[column(other + kDirectWarps)];
      double x[NT];
      load_x(col, x);
      double2 seed = seeds[32 * (int64_t)other], f = load_first(other);
      for (int cg = other; cg < ncg; cg += kDirectWarps) {
        const DevDirectCol after = cols[column(cg + 2 * kDirectWarps)];
        double xn[NT];
        load_x(next, xn);
        const double2 fn = load_first(cg + kDirectWarps);
        double2 seedn = seed;
        if (cg + kDirectWarps < ncg) seedn = seeds[32 * (int64_t)(cg + kDirectWarps)];
        const bool live = 4 * cg + t < T.nact;
        const bool dense = live && (col.row & kDirectDense) && col.start < r0 + S;
        if (dense || (live && col.start > r0 && col.start < r0 + S)) seed = make_double2(0.0, 0.0);
        const int k0 = live ? col.start - r0 : INT_MAX - 1;
        if (!__any_sync(0xffffffffu, dense)) {
          multiply(col.x2, seed, x, [&](int i, double y) { return i == k0 ? f.x : i == k0 + 1 ? f.y : y; });
        } else {
          const double *inj = p.inj + kDirectInj * (G.cols + column(cg));
          multiply(col.x2, seed, x, [&](int i, double y) {
            const int k = i - k0;
            return (dense ? k >= 0 && k < kDirectInj : k == 0 || k == 1) ? inj[k] : y;
          });
        }
        col = next;
        next = after;
        seed = seedn;
        f = fn;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) x[nt] = xn[nt];
      }
    }
    double *dst = p.alm_out + (alm_row0(M, p.lmax) + 2 * (int64_t)(G.rs + T.row0)) * p.nvecs + v0;
    const int nr = min(8 * S, R - T.row0);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (8 * nt < vn) {
        if (nt) __syncthreads();
#pragma unroll
        for (int i = 0; i < kDirectSeg; ++i)
          if (i < S)
            *reinterpret_cast<double2 *>(&s_red[warp][8 * i + g][2 * t]) = make_double2(acc[i][nt][0], acc[i][nt][1]);
        __syncthreads();
        for (int e = tid; e < 8 * nr; e += kDirectThr) {
          const int r = e >> 3, v = e & 7, at = 8 * (r % S) + r / S;
          if (8 * nt + v < vn) {
            double *to = dst + 2 * (int64_t)r * p.nvecs + 8 * nt + v;
            double a = ((s_red[0][at][v] + s_red[1][at][v]) + (s_red[2][at][v] + s_red[3][at][v])) *
                       p.scale[G.coef + T.row0 + r];
            if (p.backward) a = M.m ? 2.0 * a : (v & 1) ? 0.0 : a;
            *to = p.accumulate ? *to + a : a;
          }
        }
      }
    }
    __syncthreads();  // coefficients and sums are free for the next unit
  }
}

// ------------------------------------------------------------------------
// Plan creation: column data, first values and segment seeds of group columns
// first .. first + n - 1 (gcols: those), from the plan's strips and the row scales.
// ------------------------------------------------------------------------
__global__ void k_direct_setup(DirectParams p, const DevGCol *gcols, int64_t first, int64_t n, const double *f64,
                               DevDirectCol *cols, double *inj, double2 *seeds) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, gc = first + i;
  if (i >= n) return;
  int lo = 0, hi = p.ngroups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (p.groups[mid].cols <= gc) lo = mid;
    else hi = mid - 1;
  }
  const DevGroup G = p.groups[lo];
  const DevGCol C = gcols[i];
  const int R = G.nrows, c = (int)(gc - G.cols);
  const double2 *ab = p.ab + G.coef;
  const double *scale = p.scale + G.coef;
  DevDirectCol D{0.0, INT_MAX, C.row};
  double f[kDirectInj] = {};
  if (C.start < R) {
    D.start = C.start;
    if (C.kind == 0) {
      D.row |= kDirectDense;
      for (int i = 0; i < min(kDirectInj, R - C.start); ++i) f[i] = f64[C.data + i] / scale[C.start + i];
    } else {
      D.x2 = f64[C.data];
      for (int i = 0; i < 2; ++i) f[i] = f64[C.data + (i + 1) * (int64_t)C.nx] / scale[C.start + i];
      double a = f[0], b = f[1];
      int row = C.start;
      for (int j = (row + G.seg - 1) / G.seg; j * G.seg < R; ++j) {
        for (; row < j * G.seg; ++row) {
          const double y = row + 2 < R ? fma(fma(D.x2, ab[row + 2].x, ab[row + 2].y), b, -a) : 0.0;
          a = b;
          b = y;
        }
        seeds[p.tile_seeds[G.tile_b + j / 8] + 32 * (int64_t)(c >> 2) + 4 * (j & 7) + (c & 3)] = make_double2(a, b);
      }
    }
  }
  cols[gc] = D;
  for (int i = 0; i < kDirectInj; ++i) inj[kDirectInj * gc + i] = f[i];
}

}  // namespace

template <int NV>
static cudaError_t a2m(const DirectParams &p, int width, int npass, int grid, cudaStream_t st) {
  return launch_overlapped(width ? k_direct_a2m<NV, 2> : k_direct_a2m<NV, 1>, grid, kDirectThr, 0, st, p, npass);
}

cudaError_t launch_direct_a2m(DirectParams p, const DevDirectTileA *const (&tiles)[2], const int32_t (&ntiles)[2],
                              int sms, int max_ctas, cudaStream_t st) {
  // passes of at most 16 vectors (two columns' accumulators are then half of
  // a thread's registers), the narrowest width that covers them
  int npass = (p.nvecs + 15) / 16, nv = 2;
  constexpr int widths[] = {2, 4, 6, 8, 12, 16};
  for (int w : widths) {
    nv = w;
    if (w * npass >= p.nvecs) break;
  }
  // two columns per thread unless the units are too few to fill the GPU; a
  // thread of few vectors is short of parallel work sooner
  const int width = (int64_t)ntiles[1] * npass >= (nv <= 4 ? 16LL : 4LL) * sms;
  p.tiles_a = tiles[width];
  p.ntiles_a = ntiles[width];
  const int64_t units = (int64_t)p.ntiles_a * npass;
  if (units <= 0) return cudaSuccess;
  const int grid = (int)std::min<int64_t>(units, max_ctas > 0 ? max_ctas : INT_MAX);
  switch (nv) {
    case 2: return a2m<2>(p, width, npass, grid, st);
    case 4: return a2m<4>(p, width, npass, grid, st);
    case 6: return a2m<6>(p, width, npass, grid, st);
    case 8: return a2m<8>(p, width, npass, grid, st);
    case 12: return a2m<12>(p, width, npass, grid, st);
    default: return a2m<16>(p, width, npass, grid, st);
  }
}

cudaError_t launch_direct_m2a(const DirectParams &p, int max_ctas, cudaStream_t st) {
  // passes of 8 or 16 vectors: a step of a lane costs two operations for the
  // recurrence and eight per 8 vectors, so the wide pass wins unless half of
  // the last one would be padding
  const int n8 = (p.nvecs + 7) / 8, n16 = (p.nvecs + 15) / 16;
  const bool wide = n16 * 18 <= n8 * 10;
  const int npass = wide ? n16 : n8;
  const int64_t units = (int64_t)p.ntiles_b * npass;
  if (units <= 0) return cudaSuccess;
  const int grid = (int)std::min<int64_t>(units, max_ctas > 0 ? max_ctas : INT_MAX);
  return launch_overlapped(wide ? k_direct_m2a<2> : k_direct_m2a<1>, grid, kDirectThr, 0, st, p, npass);
}

cudaError_t launch_direct_setup(const DirectParams &p, const DevGCol *gcols, int64_t first, int64_t n,
                                const double *f64, DevDirectCol *cols, double *inj, double2 *seeds, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_direct_setup<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(p, gcols, first, n, f64, cols, inj, seeds);
  return cudaGetLastError();
}

}  // namespace wm
