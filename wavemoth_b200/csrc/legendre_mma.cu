// Tensor-core (FP64 DMMA, mma.sync m8n8k4) kernels of the interpolation
// levels of depth-1 matrices (see plan.h, build_fast_path).  For a root (T, B)
// pair:
//   alm2map   q[z] = sum_s W_T[z][s] X_T[s] + sum_s W_B[z][s] X_B[s]
//   map2alm   X_T[s] = sum_z W_T[z][s] q~[z]   (and B)
// where W[z][s] is the (n x k) matrix of one interpolation block with its
// filter folded in: row z is the unit vector e_s' if z is skeleton column s'
// (filter 0), else column c(z) of the interpolant (src/butterfly.c.in:222-235).
// The unit vectors' rows are copies; only the interpolants are multiplied.
//
// Fragment layout of mma.m8n8k4 .f64 (lane = 4 g + t): A (8x4, row) element
// (g, t); B (4x8, col) element (t, g); C/D (8x8) elements (g, 2t) and (g, 2t+1).
//
// Every output element has one writer and a fixed summation order, so results
// are bitwise reproducible.  k_seeds stores P at every kSeedRows-th row of
// every column once per split plan (legendre_split.cu slices P from them).
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
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

// D = A x B for rows 8 mt .. + 7 of one interpolation block: A(row, j) =
// a[row + j lda] (rows beyond `rows` repeat the last one and are not stored),
// B(j, v) the staged row b(j).  Eight steps of A are in flight at once.
template <int NT, class RowF>
__device__ __forceinline__ void level_tile(const double *a, int lda, int rows, int depth, int mt, RowF b,
                                           double (&acc)[NT][2]) {
  const int lane = threadIdx.x & 31, g4 = lane >> 2, t4 = lane & 3;
  const double *ap = a + min(8 * mt + g4, rows - 1);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) acc[nt][0] = acc[nt][1] = 0.0;
  for (int j0 = 0; j0 < depth; j0 += 32) {
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int j = j0 + 4 * i + t4;
      x[i] = j < depth ? ap[(int64_t)j * lda] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (j0 + 4 * i >= depth) break;
      const double *row = b(min(j0 + 4 * i + t4, depth - 1)) + g4;
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) dmma(acc[nt], x[i], row[8 * nt]);
    }
  }
}

// Starts the way of n doubles into the L2 cache.
__device__ __forceinline__ void prefetch_l2(const double *x, int n) {
  for (int e = 16 * threadIdx.x; e < n; e += 16 * kThr) asm volatile("prefetch.global.L2 [%0];" ::"l"(x + e));
}

// ------------------------------------------------------------------------
// alm2map level: one unit = one depth-1 root and 8 NT vectors.  q rows are the
// sum of the T and the B block's rows; a block's k skeleton rows are its X
// rows, its other n - k the interpolant (rows of the stored transpose) times
// X.  Interpolant rows are taken in storage order, so that A fragments are
// read from global memory as 64-byte runs without a look-up, and put in
// place through the row permutation when a tile is done.
//
// Bound: the latency of a root's small products (about 64 x 64 per block), so
// several CTAs per SM.  Reading W[z][s] through the row map element by element
// took 142 us at nside 256, 7 maps, every matrix with one level, this 85
// (map2alm 224 -> 84): 93 before the interpolants were started on their way
// to the L2 cache ahead of the X rows and the permutations read once (the
// same in map2alm, which has its operand's rows to wait for first, lost 4).
// ------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(kThr) k_a2m_level(FastParams p, int npass) {
  constexpr int NV = 8 * NT, VP = kLevelPitch<NT>;
  extern __shared__ double level_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g4 = lane >> 2, t4 = lane & 3;
  double *xs = level_smem, *ys = level_smem + p.max_root_k * VP;
  int32_t *sperm = reinterpret_cast<int32_t *>(ys + p.max_root_n * VP);  // T, then B
  for (int unit = blockIdx.x; unit < p.nroots * npass; unit += gridDim.x) {
    const DevRootUnit U = p.roots[unit / npass];
    const int v0 = (unit % npass) * NV, vn = min(NV, p.nvecs - v0);
    const DevMatrix M = p.mats[U.matrix];
    const DevPair P = p.pairs[U.pair];
    const double *X = p.xbuf + M.xrow * p.nvecs + v0;
    double *q = p.q + (int64_t)(2 * M.m + M.odd) * p.q_mstride + (int64_t)P.out_left * p.q_rstride + v0;
    prefetch_l2(p.f64 + P.ipT_t, (P.n - P.kT) * P.kT);
    prefetch_l2(p.f64 + P.ipB_t, (P.n - P.kB) * P.kB);
    for (int z = threadIdx.x; z < P.n; z += kThr) {
      sperm[z] = p.i32[P.permT + z];
      sperm[P.n + z] = p.i32[P.permB + z];
    }
    grid_wait();  // X, and the readers of q
    for (int e = threadIdx.x; e < (P.kT + P.kB) * NV; e += kThr) {
      const int s = e / NV, v = e % NV, row = s < P.kT ? P.inT + s : P.inB + (s - P.kT);
      xs[s * VP + v] = v < vn ? X[(int64_t)row * p.nvecs + v] : 0.0;
    }
    __syncthreads();
#pragma unroll 1
    for (int part = 0; part < 2; ++part) {
      const int k = part ? P.kB : P.kT, m = P.n - k;
      const double *xp = xs + (part ? P.kT * VP : 0), *ip = p.f64 + (part ? P.ipB_t : P.ipT_t);
      auto put = [&](int z, int v, double y) {
        double *at = ys + z * VP + v;
        *at = part ? *at + y : y;
      };
      for (int e = threadIdx.x; e < k * NV; e += kThr) put(sperm[part * P.n + e / NV], e % NV, xp[e / NV * VP + e % NV]);
      for (int mt = warp; 8 * mt < m; mt += kThr / 32) {
        double acc[NT][2];
        level_tile<NT>(ip, m, m, k, mt, [&](int j) { return xp + j * VP; }, acc);
        if (8 * mt + g4 < m) {
          const int z = sperm[part * P.n + k + 8 * mt + g4];
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            put(z, 8 * nt + 2 * t4, acc[nt][0]);
            put(z, 8 * nt + 2 * t4 + 1, acc[nt][1]);
          }
        }
      }
      __syncthreads();
    }
    for (int e = threadIdx.x; e < P.n * NV; e += kThr) {
      const int z = e / NV, v = e % NV;
      if (v < vn) q[(int64_t)z * p.q_rstride + v] = ys[z * VP + v];
    }
    __syncthreads();  // xs and ys are free for the next unit
  }
}

// ------------------------------------------------------------------------
// map2alm level: one unit = one depth-1 root and 8 NT vectors.  X_T[s] is q~
// at skeleton row s plus the interpolant's column s against the other rows
// (in storage order, through the permutation); B likewise.
// ------------------------------------------------------------------------
template <int NT>
__global__ void __launch_bounds__(kThr) k_m2a_level(FastParams p, int npass) {
  constexpr int NV = 8 * NT, VP = kLevelPitch<NT>;
  extern __shared__ double level_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g4 = lane >> 2, t4 = lane & 3;
  double *qs = level_smem;
  int32_t *sperm = reinterpret_cast<int32_t *>(level_smem + p.max_root_n * VP);  // T, then B
  for (int unit = blockIdx.x; unit < p.nroots * npass; unit += gridDim.x) {
    const DevRootUnit U = p.roots[unit / npass];
    const int v0 = (unit % npass) * NV, vn = min(NV, p.nvecs - v0);
    const DevMatrix M = p.mats[U.matrix];
    const DevPair P = p.pairs[U.pair];
    const double *q = p.q_in + (int64_t)(2 * M.m + M.odd) * p.q_mstride + (int64_t)P.out_left * p.q_rstride + v0;
    double *X = p.xbuf + M.xrow * p.nvecs + v0;
    for (int z = threadIdx.x; z < P.n; z += kThr) {
      sperm[z] = p.i32[P.permT + z];
      sperm[P.n + z] = p.i32[P.permB + z];
    }
    grid_wait();  // q~, and the readers of X
    for (int e = threadIdx.x; e < P.n * NV; e += kThr) {
      const int z = e / NV, v = e % NV;
      qs[z * VP + v] = v < vn ? q[(int64_t)z * p.q_rstride + v] : 0.0;
    }
    __syncthreads();
    const int mtT = (P.kT + 7) / 8, mtB = (P.kB + 7) / 8;
    for (int mt = warp; mt < mtT + mtB; mt += kThr / 32) {
      const bool isB = mt >= mtT;
      const int k = isB ? P.kB : P.kT, tile = isB ? mt - mtT : mt, s = 8 * tile + g4;
      const int32_t *perm = sperm + (isB ? P.n : 0);
      double acc[NT][2];
      level_tile<NT>(p.f64 + (isB ? P.ipB : P.ipT), k, k, P.n - k, tile,
                     [&](int j) { return qs + perm[k + j] * VP; }, acc);
      if (s < k) {
        double *dst = X + (int64_t)((isB ? P.inB : P.inT) + s) * p.nvecs;
        const double *skel = qs + perm[s] * VP;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const int v = 8 * nt + 2 * t4;
          if (v < vn) dst[v] = skel[v] + acc[nt][0];
          if (v + 1 < vn) dst[v + 1] = skel[v + 1] + acc[nt][1];
        }
      }
    }
    __syncthreads();  // qs is free for the next unit
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
cudaError_t launch_level_nt(bool alm2map, const FastParams &p, int max_ctas, cudaStream_t st) {
  const size_t smem = (size_t)level_smem_bytes<NT>(alm2map, p.max_root_n, p.max_root_k);
  const int npass = (p.nvecs + 8 * NT - 1) / (8 * NT);
  const int64_t units = (int64_t)p.nroots * npass;
  const int grid = (int)std::min<int64_t>(units, max_ctas > 0 ? max_ctas : INT_MAX);
  auto kernel = alm2map ? k_a2m_level<NT> : k_m2a_level<NT>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  return launch_overlapped(kernel, grid, kThr, smem, st, p, npass);
}

}  // namespace

cudaError_t launch_level(bool alm2map, const FastParams &p, int max_ctas, cudaStream_t st) {
  if (p.nroots <= 0) return cudaSuccess;
  // up to 32 vectors per pass, as few as cover them, and no more than leave
  // room for four CTAs per SM (16 maps at nside 256: 32 vectors per alm2map
  // pass, 82 KB and two CTAs, took 308 us with the residual)
  constexpr int64_t kRoom = 56 * 1024;
  if (p.nvecs > 16 && level_smem_bytes<4>(alm2map, p.max_root_n, p.max_root_k) <= kRoom)
    return launch_level_nt<4>(alm2map, p, max_ctas, st);
  if (p.nvecs > 8 && level_smem_bytes<2>(alm2map, p.max_root_n, p.max_root_k) <= kRoom)
    return launch_level_nt<2>(alm2map, p, max_ctas, st);
  return launch_level_nt<1>(alm2map, p, max_ctas, st);
}

cudaError_t launch_seeds(const FastParams &prm, cudaStream_t st) {
  if (prm.ngcols == 0) return cudaSuccess;
  const int block = 128;
  const int64_t grid = (prm.ngcols + block - 1) / block;
  k_seeds<<<(unsigned)grid, block, 0, st>>>(prm);
  return cudaGetLastError();
}

}  // namespace wm
