// Tensor-core (FP64 DMMA, mma.sync m8n8k4) kernels of the interpolation
// levels of depth-1 matrices (see plan.h, build_fast_path).  For a root (T, B)
// pair:
//   alm2map   q[z] = sum_s W_T[z][s] X_T[s] + sum_s W_B[z][s] X_B[s]
//   map2alm   X_T[s] = sum_z W_T[z][s] q~[z]   (and B)
// where W[z][s] is the (n x k) matrix of one interpolation block with its
// filter folded in: row z is the unit vector e_s' if z is skeleton column s'
// (filter 0), else column c(z) of the interpolant (src/butterfly.c.in:222-235).
//
// Fragment layout of mma.m8n8k4 .f64 (lane = 4 g + t): A (8x4, row) element
// (g, t); B (4x8, col) element (t, g); C/D (8x8) elements (g, 2t) and (g, 2t+1).
//
// Every output element has one writer and a fixed summation order, so results
// are bitwise reproducible.  k_seeds stores P at every kSeedRows-th row of
// every column once per split plan (legendre_split.cu slices P from them).
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"
#include "plan.h"

namespace wm {

namespace {

constexpr int kThr = 256;        // 8 warps

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// Recurrence step for group row r (>= start + 2) of column C.
__device__ __forceinline__ double rec_step(const double *f64, const DevGCol &C, double x2, int r,
                                           double pc, double pp) {
  const double *ab = f64 + C.aux + 3 * (int64_t)(r - C.boff - 2);
  return (x2 + ab[0]) * ab[1] * pc + ab[2] * pp;
}

// W[z][s] of one interpolation block (k skeleton columns, n rows z).
__device__ __forceinline__ double w_elem(const int32_t *map, const double *ip_t, int n, int k, int z,
                                         int s) {
  if (z >= n || s >= k) return 0.0;
  const int mt = map[z];
  if (mt < 0) return (s == -mt - 1) ? 1.0 : 0.0;
  return ip_t[mt + (int64_t)s * (n - k)];
}

// ------------------------------------------------------------------------
// alm2map level: one unit = one depth-1 root; q rows = W_T X_T + W_B X_B.
// ------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(kThr) k_a2m_level(FastParams p) {
  constexpr int VT = 8 * NT;
  constexpr int VP = VT + 8;
  extern __shared__ double xs[];  // (kT + kB rounded to 4) x VP
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g4 = lane >> 2, t4 = lane & 3;
  for (int unit = blockIdx.x; unit < p.nroots; unit += gridDim.x) {
    const DevRootUnit U = p.roots[unit];
    const DevMatrix M = p.mats[U.matrix];
    const DevPair P = p.pairs[U.pair];
    const int K = P.kT + P.kB, K4 = (K + 3) & ~3;
    const double *X = p.xbuf + M.xrow * p.nvecs;
    double *qm = p.q + (int64_t)(2 * M.m + M.odd) * p.q_mstride;
    const int32_t *mapT = p.i32 + P.mapT, *mapB = p.i32 + P.mapB;
    const double *ipT = p.f64 + P.ipT_t, *ipB = p.f64 + P.ipB_t;
    for (int v0 = 0; v0 < p.nvecs; v0 += VT) {
      const int vn = min(VT, p.nvecs - v0);
      __syncthreads();
      for (int idx = threadIdx.x; idx < K4 * VT; idx += kThr) {
        const int s = idx / VT, v = idx % VT;
        double val = 0.0;
        if (s < K && v < vn) {
          const int row = s < P.kT ? P.inT + s : P.inB + (s - P.kT);
          val = X[(int64_t)row * p.nvecs + v0 + v];
        }
        xs[s * VP + v] = val;
      }
      __syncthreads();
      for (int z0 = 0; z0 < P.n; z0 += 128) {
        double acc[2][NT][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) acc[i][nt][0] = acc[i][nt][1] = 0.0;
        for (int ks = 0; ks < K4 / 4; ++ks) {
          const int s = 4 * ks + t4;
          double a[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int z = z0 + 16 * warp + 8 * i + g4;
            a[i] = s < P.kT ? w_elem(mapT, ipT, P.n, P.kT, z, s)
                            : w_elem(mapB, ipB, P.n, P.kB, z, s - P.kT);
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const double b = xs[s * VP + 8 * nt + g4];
            dmma(acc[0][nt], a[0], b);
            dmma(acc[1][nt], a[1], b);
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int z = z0 + 16 * warp + 8 * i + g4;
          if (z >= P.n) continue;
          double *dst = qm + (int64_t)(P.out_left + z) * p.q_rstride + v0;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const int v = 8 * nt + 2 * t4;
            if (v < vn) dst[v] = acc[i][nt][0];
            if (v + 1 < vn) dst[v + 1] = acc[i][nt][1];
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------------
// map2alm level: one unit = one depth-1 root; X_T = W_T^T q~, X_B = W_B^T q~.
// ------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(kThr) k_m2a_level(FastParams p) {
  constexpr int VT = 8 * NT;
  constexpr int VP = VT + 8;
  extern __shared__ double qs[];  // (n rounded to 4) x VP
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g4 = lane >> 2, t4 = lane & 3;
  for (int unit = blockIdx.x; unit < p.nroots; unit += gridDim.x) {
    const DevRootUnit U = p.roots[unit];
    const DevMatrix M = p.mats[U.matrix];
    const DevPair P = p.pairs[U.pair];
    const int n4 = (P.n + 3) & ~3;
    const double *qm = p.q_in + (int64_t)(2 * M.m + M.odd) * p.q_mstride;
    double *X = p.xbuf + M.xrow * p.nvecs;
    const int mtT = (P.kT + 7) / 8, mtB = (P.kB + 7) / 8, mtiles = mtT + mtB;
    for (int v0 = 0; v0 < p.nvecs; v0 += VT) {
      const int vn = min(VT, p.nvecs - v0);
      __syncthreads();
      for (int idx = threadIdx.x; idx < n4 * VT; idx += kThr) {
        const int z = idx / VT, v = idx % VT;
        double val = 0.0;
        if (z < P.n && v < vn) val = qm[(int64_t)(P.out_left + z) * p.q_rstride + v0 + v];
        qs[z * VP + v] = val;
      }
      __syncthreads();
      for (int mt = warp; mt < mtiles; mt += kThr / 32) {
        const bool isB = mt >= mtT;
        const int k = isB ? P.kB : P.kT;
        const int s = (isB ? mt - mtT : mt) * 8 + g4;
        const int32_t *map = p.i32 + (isB ? P.mapB : P.mapT);
        const double *ipt = p.f64 + (isB ? P.ipB_t : P.ipT_t);
        double acc[NT][2];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
        for (int ks = 0; ks < n4 / 4; ++ks) {
          const int z = 4 * ks + t4;
          const double a = w_elem(map, ipt, P.n, k, z, s);
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) dmma(acc[nt], a, qs[(4 * ks + t4) * VP + 8 * nt + g4]);
        }
        if (s < k) {
          double *dst = X + (int64_t)((isB ? P.inB : P.inT) + s) * p.nvecs + v0;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const int v = 8 * nt + 2 * t4;
            if (v < vn) dst[v] = acc[nt][0];
            if (v + 1 < vn) dst[v + 1] = acc[nt][1];
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------------
// Seeds: P at rows (s, s + 1), s = max(chunk start, column start), for every
// recurrence column and row chunk of its group.
// ------------------------------------------------------------------------
__global__ void k_seeds(FastParams p) {
  const int64_t gc = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (gc >= p.ngcols) return;
  // locate the group (binary search over group column offsets)
  int lo = 0, hi = p.ngroups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (p.groups[mid].cols <= gc) lo = mid; else hi = mid - 1;
  }
  const DevGroup G = p.groups[lo];
  const int c = (int)(gc - G.cols);
  const DevGCol C = p.gcols[gc];
  double *seed = p.seeds_out + G.seeds + (int64_t)c * G.nchunks * 2;
  for (int j = 0; j < G.nchunks; ++j) {
    seed[2 * j] = 0.0;
    seed[2 * j + 1] = 0.0;
  }
  if (C.kind != 1 || C.start >= G.nrows) return;
  const double x2 = p.f64[C.data];
  double a = p.f64[C.data + C.nx], b = p.f64[C.data + 2 * C.nx];  // P[row], P[row + 1]
  int row = C.start;
  for (int j = 0; j < G.nchunks; ++j) {
    const int target = max(j * kSeedRows, C.start);
    if (target >= G.nrows) break;
    while (row < target) {
      // P[row + 2] exists only inside the group's rows
      const double nv = (row + 2 < G.nrows) ? rec_step(p.f64, C, x2, row + 2, b, a) : 0.0;
      a = b;
      b = nv;
      ++row;
    }
    seed[2 * j] = a;
    seed[2 * j + 1] = b;
  }
}

template <int NT>
cudaError_t launch_nt(int which, const FastParams &prm, int grid, size_t smem, cudaStream_t st) {
  switch (which) {
    case 1: {
      cudaError_t e = cudaFuncSetAttribute(k_a2m_level<NT>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      k_a2m_level<NT><<<grid, kThr, smem, st>>>(prm);
      break;
    }
    case 2: {
      cudaError_t e = cudaFuncSetAttribute(k_m2a_level<NT>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      k_m2a_level<NT><<<grid, kThr, smem, st>>>(prm);
      break;
    }
  }
  return cudaGetLastError();
}

}  // namespace

int fast_vector_tiles(int nvecs) {
  // N-tiles of 8 vectors per pass: the smallest power of two covering
  // nvecs, at most 8 (64 vectors per pass)
  int nt = 1;
  while (nt < 8 && 8 * nt < nvecs) nt *= 2;
  return nt;
}

cudaError_t launch_fast(int which, const FastParams &prm, int grid, cudaStream_t st) {
  const int NT = fast_vector_tiles(prm.nvecs);
  const int VP = 8 * NT + 8;
  size_t smem = 0;
  if (which == 1) smem = (size_t)((prm.max_root_k + 3) & ~3) * VP * sizeof(double);
  if (which == 2) smem = (size_t)((prm.max_root_n + 3) & ~3) * VP * sizeof(double);
  if (which == 1 || which == 2) smem = smem < 16 ? 16 : smem;
  switch (NT) {
    case 1: return launch_nt<1>(which, prm, grid, smem, st);
    case 2: return launch_nt<2>(which, prm, grid, smem, st);
    case 4: return launch_nt<4>(which, prm, grid, smem, st);
    default: return launch_nt<8>(which, prm, grid, smem, st);
  }
}

cudaError_t launch_seeds(const FastParams &prm, cudaStream_t st) {
  if (prm.ngcols == 0) return cudaSuccess;
  const int block = 128;
  const int64_t grid = (prm.ngcols + block - 1) / block;
  k_seeds<<<(unsigned)grid, block, 0, st>>>(prm);
  return cudaGetLastError();
}

}  // namespace wm
