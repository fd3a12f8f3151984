// C ABI of libwavemoth_b200.so: the plan object and every extern "C" entry
// point declared in include/wavemoth.h and include/wavemoth_b200.h.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <sys/stat.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <tuple>
#include <vector>

#include "kernels.h"
#include "plan.h"
#include "program.h"
#include "wavemoth.h"
#include "wavemoth_b200.h"

namespace {

thread_local std::string g_last_error;
std::string g_resource_dir;
int64_t g_device_cap = 0;

int set_error(int code, const std::string &msg) {
  g_last_error = msg;
  return code;
}

struct DeviceArena {
  std::vector<void *> ptrs;
  int64_t bytes = 0;
  int64_t base = 0;  // bytes held elsewhere on behalf of the same plan (its shared image)
  ~DeviceArena() {
    for (void *p : ptrs) cudaFree(p);
  }
  template <class T>
  int alloc(T **out, size_t count, const char *what) {
    size_t nbytes = std::max<size_t>(count, 1) * sizeof(T);
    if (g_device_cap > 0 && base + bytes + (int64_t)nbytes > g_device_cap)
      return set_error(WAVEMOTH_ERR_NOMEM, std::string("device memory cap exceeded allocating ") + what);
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, nbytes);
    if (e != cudaSuccess)
      return set_error(WAVEMOTH_ERR_NOMEM, std::string("cudaMalloc(") + what + "): " +
                                               cudaGetErrorString(e));
    ptrs.push_back(p);
    bytes += (int64_t)nbytes;
    *out = (T *)p;
    return 0;
  }
  // Takes over the allocations of another arena.
  void adopt(DeviceArena &other) {
    ptrs.insert(ptrs.end(), other.ptrs.begin(), other.ptrs.end());
    bytes += other.bytes;
    other.ptrs.clear();
    other.bytes = 0;
  }
};

}  // namespace

// Device data of a compiled plan file that does not depend on the number of
// maps: the butterfly program, the tables of the FP64 and of the split path,
// the ring tables, the sliced P and W.  Read-only once built; what only some
// plans of a split image read (the FP64 tables, the sliced P) is added when the
// first of them is made, and plans see what there was when they were made.
struct ImageRefs {
  wm::DevMatrix *d_mats = nullptr;
  wm::DevDBlock *d_dblocks = nullptr;
  wm::DevStrip *d_strips = nullptr;
  wm::DevLevel *d_levels = nullptr;
  wm::DevPair *d_pairs = nullptr;
  double *d_f64 = nullptr;
  int32_t *d_i32 = nullptr;
  int32_t *d_order = nullptr;       // all matrices, largest first (generic kernel over everything)
  int32_t *d_order_slow = nullptr;  // matrices left to the generic kernel (build_fast_path)
  int32_t nslow = 0;
  // row groups
  wm::DevGroup *d_groups = nullptr;
  wm::DevGCol *d_gcols = nullptr;
  wm::DevRootUnit *d_roots = nullptr;
  // FP64 residual path
  bool direct = false;
  const wm::DevDirectTileA *d_direct_a[2] = {};
  int32_t ndirect_a[2] = {};
  wm::DevDirectTileB *d_direct_b = nullptr;
  int32_t ndirect_b = 0;
  double *d_direct_ab = nullptr, *d_direct_scale = nullptr, *d_direct_inj = nullptr;
  wm::DevDirectCol *d_direct_cols = nullptr;
  double2 *d_direct_seeds = nullptr;
  int64_t *d_direct_tile_seeds = nullptr;
  // split-precision path
  bool split = false;
  double *d_seeds = nullptr;
  wm::DevSplitGroup *d_sgroups = nullptr;
  wm::DevSplitTileA *d_stiles_a = nullptr;
  wm::DevSplitTileB *d_stiles_b = nullptr;
  double2 *d_col_scale = nullptr, *d_row_scale = nullptr;
  wm::DevSplitRoot *d_sroots = nullptr;
  wm::DevSplitLevelTile *d_stiles_la = nullptr, *d_stiles_lm = nullptr;
  int8_t *d_level_a = nullptr;
  double2 *d_level_rs = nullptr;
  // streamed split GEMM launches (wm::kStream*) and the residual P sliced
  // once per image (null: generated by the GEMM kernels at every call)
  wm::DevStreamTile *d_stream_tiles[4] = {};
  int32_t *d_stream_rows[4] = {}, *d_stream_sidx[4] = {};
  int32_t nstream[4] = {};
  int64_t *d_split_zero[4] = {};   // rows no split tile writes (per launch), zeroed before it
  int32_t nsplit_zero[4] = {};
  int8_t *d_res_a = nullptr;
  int64_t res_a_bytes = 0;
  // rings
  wm::DevRing *d_rings = nullptr;
  int32_t *d_ring_mend = nullptr;  // per ring pair: the synthesis gather's m limit (HostProgram::ring_mend)
  double2 *d_phases = nullptr;  // per ring pair: e^{i m phi0}, fine and coarse tables
  double *d_twiddles = nullptr, *d_filters = nullptr, *d_ring_aux = nullptr;
  int32_t twlen = 0, max_bluestein = 0, nphase_hi = 1;
};

struct DeviceImage : ImageRefs {
  DeviceArena arena;
  wm::HostProgram prog;
  int64_t program_bytes = 0;
  std::vector<int64_t> m_bounds;  // m-sharded images: every part's m range
};

struct _wavemoth_plan : ImageRefs {
  int nside = 0, lmax = 0, mmax = 0, nmaps = 0, nvecs = 0, ni = 0;
  int64_t npix = 0, nalm = 0;
  unsigned flags = 0;
  bool analysis = false;          // map2alm plan
  double *host_in = nullptr, *host_out = nullptr;
  int status = 0;
  int phase_shifts = 1;
  int64_t wait_limit = 0;         // streamed split GEMM waits (0: the kernel's default)
  int grid_cap = 0;               // SMs for the persistent Legendre kernels (0: all)
  // m-sharded plans: part `part` of `nparts`, the parts' m and ring-pair ranges
  int nparts = 1, part = 0;
  std::vector<int64_t> m_bounds, ring_bounds;
  int64_t *d_shard_tab = nullptr;
  int sm_count = 0;
  int grid = 0;
  std::string resource_path;      // the plan file (empty for dense-recurrence plans)

  // the shared image (plans of one file, lmax, mmax and precision share it)
  // and this plan's own per-call buffers
  std::shared_ptr<DeviceImage> img;
  DeviceArena arena;
  int32_t *d_counter = nullptr;
  double *d_xbuf = nullptr;
  double2 *d_vec_scale = nullptr;
  int8_t *d_planes = nullptr;
  int32_t *d_status = nullptr;
  wm::DevRingTask *d_ring_tasks = nullptr;
  int32_t ring_ntasks = 0, ring_smem = 0, ring_threads = 0, ring_short = 0;
  double *d_alm = nullptr, *d_map = nullptr, *d_q = nullptr, *d_scratch = nullptr;
  double *d_ring_weights = nullptr;           // per ring pair (null: unweighted analysis)
  double *d_ring_weights_buf = nullptr;
  double *d_iter_map = nullptr, *d_iter_alm = nullptr;  // iterative map2alm buffers (on first use)
  int64_t slot_stride = 0;
  cudaStream_t stream = nullptr;

  // optional per-kernel event timing (wavemoth_plan_timing)
  bool timing = false;
  // kernels launched by executes since the last timing reset
  int64_t kernel_launches = 0;
  struct Span { int kind; cudaEvent_t a, b; };
  std::vector<Span> spans;

  ~_wavemoth_plan() {
    for (auto &s : spans) { cudaEventDestroy(s.a); cudaEventDestroy(s.b); }
    if (stream) cudaStreamDestroy(stream);
  }
};

namespace {

// m values in the plan's q: all of them, or the shard's own
int64_t shard_mcount(wavemoth_plan P) {
  return P->nparts > 1 ? P->m_bounds[P->part + 1] - P->m_bounds[P->part] : (int64_t)P->mmax + 1;
}

int cuda_check(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return 0;
  return set_error(WAVEMOTH_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

template <class T>
int upload(DeviceArena &A, T **dst, const std::vector<T> &src, const char *what) {
  if (int rc = A.alloc(dst, src.size(), what)) return rc;
  if (!src.empty())
    return cuda_check(cudaMemcpy(*dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice),
                      what);
  return 0;
}

bool read_file(const std::string &path, std::vector<char> &buf, std::string &err) {
  FILE *f = fopen(path.c_str(), "rb");
  if (!f) {
    err = "cannot open resource file " + path;
    return false;
  }
  fseek(f, 0, SEEK_END);
  long n = ftell(f);
  fseek(f, 0, SEEK_SET);
  if (n < 0) {
    fclose(f);
    err = "cannot size resource file " + path;
    return false;
  }
  buf.resize((size_t)n);
  size_t got = n ? fread(buf.data(), 1, (size_t)n, f) : 0;
  fclose(f);
  if (got != (size_t)n) {
    err = "short read of resource file " + path;
    return false;
  }
  return true;
}

struct RingTable {
  std::vector<wm::DevRing> rings;
  std::vector<wm::DevRingTask> tasks;  // by decreasing cost
  int64_t filter_cplx = 0;   // complex entries of all Bluestein filter spectra
  int64_t aux_cplx = 0;      // complex entries of all Bluestein chirp/root tables
  int32_t twlen = 4;         // largest power-of-two table length needed
  int32_t max_bluestein = 0;
  int32_t smem = 0;
  int32_t threads = 0, short_rings = 0;
  int32_t nphase_hi = 1;
  int64_t max_cta_cplx = 0;  // largest transform buffer of one CTA
};

// Ring geometry (src/wavemoth.c:1199-1232) and the CTA work list of the ring
// kernels: per ring pair, groups of G maps with both hemispheres and
// 2 G x (transform length) within the CTA buffer; transforms longer than half
// the buffer run one map and one hemisphere per CTA.  Ordered by decreasing
// cost so that the long transforms start first.
RingTable ring_table(int nside, int nmaps, int mmax, bool one_side = false) {
  const int nrings = 4 * nside - 1, mid = 2 * nside - 1;
  std::vector<int64_t> offs(nrings + 1);
  int64_t ipix = 0, npr = 0;
  std::vector<int> num(nrings), den(nrings);
  for (int r = 0; r < nrings; ++r) {
    if (r <= nside - 1) {
      npr += 4;
      num[r] = 1;
      den[r] = 4 * (r + 1);
    } else if (r > 3 * nside - 1) {
      npr -= 4;
      num[r] = 1;
      den[r] = 4 * (nrings - r);
    } else {
      num[r] = r % 2;
      den[r] = 4 * nside;
    }
    offs[r] = ipix;
    ipix += npr;
  }
  offs[nrings] = ipix;
  RingTable T;
  T.rings.resize(2 * nside);
  T.nphase_hi = mmax / 64 + 1;
  int gmax = 1;
  while (gmax < nmaps && gmax < 8) gmax <<= 1;
  // longest transform of one map, both hemispheres, and from it the transform
  // buffer of a CTA: as small as holds it, so that several CTAs per SM hide
  // one another's global reads and barriers.  Large batches take twice that:
  // the groups of maps that read a q row together are wider.  Measured,
  // synthesis + analysis, buffer of 2048 / 4096 / 8192 points (CTAs of 128 /
  // 256 / 512 threads): nside 256 (2048 points per map), 1 map 52 / 84 / 126
  // us, 16 maps 370 / 352 / 372, 32 maps 705 / 640 / 681; nside 512 (4096),
  // 1 map - / 153 / 215 us, 3 maps - / 371 / 389, 16 maps - / 1439 / 1355;
  // nside 1024 (8192) has no choice.
  int longest = 1;
  for (int r = 0; r < 2 * nside; ++r) {
    const int N = (int)(offs[mid + r + 1] - offs[mid + r]) / 2;
    int len = 1;
    while (len < ((N & (N - 1)) ? 2 * N - 1 : N)) len <<= 1;
    longest = std::max(longest, 2 * len);
  }
  //
  // The shortest rings (up to nside 64; by the ring length alone, so that a map
  // gives the same bits whatever is beside it) run in passes of radix 4: a
  // radix-16 butterfly of theirs keeps one thread busy for longer than the
  // passes it saves take.  A quarter of the points per CTA then feed every
  // thread; with 16 maps and more, as many as before.  Measured, alm2map /
  // map2alm, radix 16 -> 4, us: nside 32, 3 maps 14.3 / 12.6 -> 14.0 / 10.4, 32
  // maps 23.2 / 22.1 -> 23.6 / 19.9; nside 64, 1 map 15.3 / 15.4 -> 14.9 / 11.2, 8
  // maps 20.1 / 20.0 -> 19.6 / 17.8, 32 maps 43.8 / 43.4 -> 44.9 / 43.1; nside
  // 256, 1 map 56 / 100 -> 60 / 103.
  const bool short_rings = longest <= 512;
  const int least = short_rings ? 512 : 2048, most = short_rings ? 4 * longest : 2 * longest;
  const int buffer = std::min(wm::kRingBufferCplx, std::max(least, nmaps >= 16 ? most : longest));
  struct Item { double cost; wm::DevRingTask t; int64_t cplx; };
  std::vector<Item> items;
  for (int r = 0; r < 2 * nside; ++r) {
    wm::DevRing R{};
    R.n = (int32_t)(offs[mid + r + 1] - offs[mid + r]);
    R.phi_num = num[mid + r];
    R.phi_den = den[mid + r];
    R.off_north = offs[mid - r];
    R.off_south = offs[mid + r];
    const int N = R.n / 2;
    int len = N;
    if (N & (N - 1)) {
      int M = 1;
      while (M < 2 * N - 1) M <<= 1;
      R.bluestein_m = M;
      R.filter = T.filter_cplx;
      T.filter_cplx += M;
      R.aux = T.aux_cplx;
      T.aux_cplx += 2 * N + 1;
      T.max_bluestein = std::max(T.max_bluestein, M);
      len = M;
      T.twlen = std::max(T.twlen, M);
    } else {
      T.twlen = std::max(T.twlen, 2 * N);  // roots e^{2 pi i k / n}, n = 2N
    }
    T.rings[r] = R;
    // both hemispheres in one CTA (lanes = sides x maps) when they fit the
    // buffer; the longest transforms run one hemisphere at a time
    int G = 1, two = 1;
    if (one_side) {
      two = 0;
      G = std::max(1, std::min(gmax, wm::kRingBufferCplx / len));
    } else if (2 * len <= wm::kRingBufferCplx) {
      G = std::min(gmax, std::max(1, buffer / (2 * len)));
    } else {
      two = 0;
    }
    int lg = 0;
    while ((1 << lg) < G) ++lg;
    const int64_t cplx = (int64_t)G * len << two;
    const double cost = (double)cplx * (R.bluestein_m ? 2.5 : 1.0) + (double)G * (mmax + 1);
    T.max_cta_cplx = std::max(T.max_cta_cplx, cplx);
    for (int g0 = 0; g0 < nmaps; g0 += G)
      items.push_back({cost, wm::DevRingTask{r, g0, lg, two}, cplx});
  }
  std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) { return a.cost > b.cost; });
  int64_t need = 0;
  for (const Item &it : items) {
    T.tasks.push_back(it.t);
    need = std::max(need, it.cplx);
  }
  T.smem = T.tasks.empty() ? 0 : wm::ring_cta_smem(need, T.nphase_hi);
  T.threads = need > 4096 ? 512 : need > 2048 ? 256 : 128;  // 16 points per thread
  T.short_rings = short_rings;
  return T;
}

wm::RingParams ring_params(wavemoth_plan P);
wm::StreamLaunch stream_launch(wavemoth_plan P, int k);

wm::FastParams fast_params(wavemoth_plan P) {
  const auto &G = P->img->prog;
  wm::FastParams f{};
  f.mats = P->d_mats;
  f.pairs = P->d_pairs;
  f.f64 = P->d_f64;
  f.i32 = P->d_i32;
  f.groups = P->d_groups;
  f.gcols = P->d_gcols;
  f.roots = P->d_roots;
  f.ngroups = (int32_t)G.groups.size();
  f.ngcols = G.ngcols;
  f.nroots = (int32_t)G.roots.size();
  f.max_root_k = G.max_root_k;
  f.max_root_n = G.max_root_n;
  f.nvecs = P->nvecs;
  f.q_mstride = P->nvecs;
  f.q_rstride = 2LL * shard_mcount(P) * P->nvecs;
  f.xbuf = P->d_xbuf;
  return f;
}

wm::DirectParams direct_params(wavemoth_plan P) {
  wm::DirectParams d{};
  d.mats = P->d_mats;
  d.groups = P->d_groups;
  d.cols = P->d_direct_cols;
  d.inj = P->d_direct_inj;
  d.ab = reinterpret_cast<const double2 *>(P->d_direct_ab);
  d.scale = P->d_direct_scale;
  d.seeds = P->d_direct_seeds;
  d.tile_seeds = P->d_direct_tile_seeds;
  d.tiles_b = P->d_direct_b;
  d.ntiles_b = P->ndirect_b;
  d.ngroups = (int32_t)P->img->prog.groups.size();
  d.ngcols = P->img->prog.ngcols;
  d.lmax = P->lmax;
  d.nvecs = P->nvecs;
  d.q_mstride = P->nvecs;
  d.q_rstride = 2LL * shard_mcount(P) * P->nvecs;
  d.xbuf = P->d_xbuf;
  return d;
}

wm::SplitParams split_params(wavemoth_plan P) {
  const auto &G = P->img->prog;
  wm::SplitParams s{};
  s.mats = P->d_mats;
  s.f64 = P->d_f64;
  s.groups = P->d_groups;
  s.gcols = P->d_gcols;
  s.sgroups = P->d_sgroups;
  s.tiles_a = P->d_stiles_a;
  s.tiles_b = P->d_stiles_b;
  s.ngroups = (int32_t)G.groups.size();
  s.ngcols = G.ngcols;
  s.ntiles_a = (int32_t)G.stiles_a.size();
  s.ntiles_b = (int32_t)G.stiles_b.size();
  s.seeds = P->d_seeds;
  s.col_scale = P->d_col_scale;
  s.row_scale = P->d_row_scale;
  s.vec_scale = P->d_vec_scale;
  s.planes = P->d_planes;
  s.nrowscale = G.split_rows;
  s.lmax = P->lmax;
  s.nvecs = P->nvecs;
  s.ni = P->ni;
  s.q_mstride = P->nvecs;
  s.q_rstride = 2LL * shard_mcount(P) * P->nvecs;
  s.xbuf = P->d_xbuf;
  s.status = P->d_status;
  s.wait_limit = P->wait_limit;
  s.pairs = P->d_pairs;
  s.i32 = P->d_i32;
  s.roots = P->d_roots;
  s.sroots = P->d_sroots;
  s.tiles_la = P->d_stiles_la;
  s.tiles_lm = P->d_stiles_lm;
  s.nroots = (int32_t)G.roots.size();
  s.ntiles_la = (int32_t)G.stiles_la.size();
  s.ntiles_lm = (int32_t)G.stiles_lm.size();
  s.level_a = P->d_level_a;
  s.level_rs = P->d_level_rs;
  return s;
}

// Whether a split plan's number of maps puts its Legendre step on the FP64
// units, on images large enough (kDirectMinElems) whose roots the level kernels
// hold.  The split GEMMs stream six bytes of sliced P per element whatever the
// number of maps, the FP64 kernels do two operations and one per vector.
// Measured, alm2map + map2alm, FP64 / split, us: nside 128, lmax 256: 3 maps 43
// / 130, 16 maps 106 / 138; nside 256, lmax 512: 8 maps 284 / 485, 16 maps 500 /
// 507; nside 512, lmax 1024: 8 maps 1501 / 2261, 16 maps 2861 / 2330; nside 1024,
// lmax 1500: 3 maps 2841 / 7254, 8 maps 5474 / 7532, 16 maps 10660 / 7838.  Plans
// that are to generate P rather than hold it would hold the FP64 tables instead,
// and keep the GEMMs.
// kDirectMinElems is not where the times cross.  FP64 is the faster one below it
// as well (1 / 4 / 14 maps: nside 32, lmax 64 21 / 23 / 27 us against 50 / 51 / 55;
// nside 64, lmax 191 31 / 37 / 73 against 78 / 83 / 97; nside 96, lmax 192 39 / 50 /
// 116 against 105 / 111 / 165); the bound leaves split plans of small files the
// kernels, and the bits, that they have always had.
constexpr int64_t kDirectMinElems = 4 << 20;

bool prefers_direct(wavemoth_plan P) {
  const auto &G = P->img->prog;
  if ((P->flags & WAVEMOTH_SPLIT_GENERATE) || G.rec_elems < kDirectMinElems ||
      !wm::level_fits(G.max_root_n, G.max_root_k))
    return false;
  return P->nvecs <= (G.rec_elems + G.interp_elems <= 80000000 ? 28 : 16);
}

// Whether a plan's Legendre step runs on the FP64 units: always without split
// precision, and with it where that is preferred and the image has the tables.
// A plan with a wait limit set keeps the kernels whose waits it bounds.
bool use_direct(wavemoth_plan P) {
  return !P->split || (P->direct && P->wait_limit == 0 && prefers_direct(P));
}

// Images of compiled plan files, shared by the plans that use the same file
// (path, size, modification time), lmax, mmax and precision flags; an image
// lives as long as one of its plans.  Plan creation is serialised.
struct ImageKey {
  std::string path;
  int64_t size, mtime;
  int lmax, mmax;
  unsigned flags;
  int nparts, part;  // m-sharded images hold one part's tables
  bool operator<(const ImageKey &o) const {
    return std::tie(path, size, mtime, lmax, mmax, flags, nparts, part) <
           std::tie(o.path, o.size, o.mtime, o.lmax, o.mmax, o.flags, o.nparts, o.part);
  }
};
std::mutex g_image_mutex;
std::map<ImageKey, std::weak_ptr<DeviceImage>> g_images;

// Tables of the FP64 residual path, allocated in A (setup_direct fills them).
int build_direct(ImageRefs &I, const wm::HostProgram &G, DeviceArena &A) {
  const size_t nc = (size_t)G.ngcols;
  int rc = 0;
  for (int w = 0; w < 2; ++w) {
    wm::DevDirectTileA *tiles = nullptr;
    rc = rc ? rc : upload(A, &tiles, G.direct_a[w], "alm2map tiles");
    I.d_direct_a[w] = tiles;
    I.ndirect_a[w] = (int32_t)G.direct_a[w].size();
  }
  rc = rc ? rc : upload(A, &I.d_direct_b, G.direct_b, "map2alm tiles");
  I.ndirect_b = (int32_t)G.direct_b.size();
  rc = rc ? rc : upload(A, &I.d_direct_tile_seeds, G.direct_tile_seeds, "seed tables");
  rc = rc ? rc : upload(A, &I.d_direct_ab, G.direct_ab, "row coefficients");
  rc = rc ? rc : upload(A, &I.d_direct_scale, G.direct_scale, "row scales");
  rc = rc ? rc : A.alloc(&I.d_direct_cols, nc, "column table");
  rc = rc ? rc : A.alloc(&I.d_direct_inj, nc * wm::kDirectInj, "column first values");
  rc = rc ? rc : A.alloc(&I.d_direct_seeds, (size_t)G.direct_seeds, "segment seeds");
  I.direct = rc == 0;
  return rc;
}

// Uploads the map-count independent tables of `img` (whose program is
// compiled) and allocates its plan-time outputs; the plan-time kernels run
// later, through the first plan.
int build_image(DeviceImage &I, int nside, int mmax, unsigned flags) {
  auto &G = I.prog;
  DeviceArena &A = I.arena;
  int rc = 0;
  std::vector<int32_t> order(G.mats.size());
  std::iota(order.begin(), order.end(), 0);
  if (G.shard_m1 >= 0)  // a shard's generic kernel sees its own matrices only
    order.erase(std::remove_if(order.begin(), order.end(),
                               [&](int i) { return G.mats[i].m < G.shard_m0 || G.mats[i].m >= G.shard_m1; }),
                order.end());
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return G.mats[a].cost > G.mats[b].cost; });
  rc = rc ? rc : upload(A, &I.d_mats, G.mats, "matrices");
  rc = rc ? rc : upload(A, &I.d_dblocks, G.dblocks, "residual blocks");
  rc = rc ? rc : upload(A, &I.d_strips, G.strips, "strips");
  rc = rc ? rc : upload(A, &I.d_levels, G.levels, "levels");
  rc = rc ? rc : upload(A, &I.d_pairs, G.pairs, "pairs");
  rc = rc ? rc : upload(A, &I.d_f64, G.f64, "f64 arena");
  rc = rc ? rc : upload(A, &I.d_i32, G.i32, "i32 arena");
  rc = rc ? rc : upload(A, &I.d_order, order, "order");
  {
    std::vector<int32_t> slow;
    std::vector<char> is_slow(G.mats.size(), 0);
    for (int32_t mi : G.slow_mats) is_slow[mi] = 1;
    for (int32_t mi : order)
      if (is_slow[mi]) slow.push_back(mi);
    I.nslow = (int32_t)slow.size();
    rc = rc ? rc : upload(A, &I.d_order_slow, slow, "slow order");
  }
  rc = rc ? rc : upload(A, &I.d_groups, G.groups, "groups");
  // (the FP64 path's tables are made from the group columns and replace them)
  if (flags & WAVEMOTH_PRECISION_SPLIT) rc = rc ? rc : upload(A, &I.d_gcols, G.gcols, "group columns");
  rc = rc ? rc : upload(A, &I.d_roots, G.roots, "roots");
  I.split = (flags & WAVEMOTH_PRECISION_SPLIT) != 0;
  if (!I.split) rc = rc ? rc : build_direct(I, G, A);
  if (I.split) rc = rc ? rc : A.alloc(&I.d_seeds, (size_t)std::max<int64_t>(G.nseeds, 1), "recurrence seeds");
  I.program_bytes = A.bytes;
  {
    RingTable RT = ring_table(nside, 1, mmax);
    I.twlen = RT.twlen;
    I.max_bluestein = RT.max_bluestein;
    I.nphase_hi = RT.nphase_hi;
    rc = rc ? rc : upload(A, &I.d_rings, RT.rings, "ring table");
    if (!G.ring_mend.empty()) rc = rc ? rc : upload(A, &I.d_ring_mend, G.ring_mend, "ring m limits");
    rc = rc ? rc : A.alloc(&I.d_twiddles, (size_t)RT.twlen, "twiddle table");
    rc = rc ? rc : A.alloc(&I.d_filters, (size_t)std::max<int64_t>(2 * RT.filter_cplx, 2), "Bluestein filters");
    rc = rc ? rc : A.alloc(&I.d_ring_aux, (size_t)std::max<int64_t>(2 * RT.aux_cplx, 2), "Bluestein chirps");
    rc = rc ? rc : A.alloc(&I.d_phases, (size_t)(2 * nside) * (wm::kRingPhaseLo + RT.nphase_hi), "phase tables");
  }
  if (I.split) {
    rc = rc ? rc : upload(A, &I.d_sgroups, G.sgroups, "split groups");
    rc = rc ? rc : upload(A, &I.d_stiles_a, G.stiles_a, "split alm2map tiles");
    rc = rc ? rc : upload(A, &I.d_stiles_b, G.stiles_b, "split map2alm tiles");
    rc = rc ? rc : A.alloc(&I.d_col_scale, (size_t)std::max<int64_t>((int64_t)G.gcols.size(), 1), "column scales");
    rc = rc ? rc : A.alloc(&I.d_row_scale, (size_t)std::max<int64_t>(G.split_rows, 1), "row scales");
    rc = rc ? rc : upload(A, &I.d_sroots, G.sroots, "split roots");
    rc = rc ? rc : upload(A, &I.d_stiles_la, G.stiles_la, "split alm2map level tiles");
    rc = rc ? rc : upload(A, &I.d_stiles_lm, G.stiles_lm, "split map2alm level tiles");
    rc = rc ? rc : A.alloc(&I.d_level_a,
                           (size_t)std::max<int64_t>(G.split_level_blocks, 1) * wm::kSplitBlock,
                           "sliced interpolation matrices");
    rc = rc ? rc : A.alloc(&I.d_level_rs, (size_t)std::max<int64_t>(G.split_level_rows, 1),
                           "interpolation row scales");
    for (int k = 0; k < 4; ++k) {
      rc = rc ? rc : upload(A, &I.d_stream_tiles[k], G.stream_tiles[k], "streamed GEMM tiles");
      rc = rc ? rc : upload(A, &I.d_stream_rows[k], G.stream_rows[k], "streamed GEMM rows");
      rc = rc ? rc : upload(A, &I.d_stream_sidx[k], G.stream_sidx[k], "streamed GEMM scales");
      I.nstream[k] = (int32_t)G.stream_tiles[k].size();
      rc = rc ? rc : upload(A, &I.d_split_zero[k], G.split_zero[k], "split zero rows");
      I.nsplit_zero[k] = (int32_t)G.split_zero[k].size();
    }
  }
  return rc;
}

// Whether `need` more bytes fit beside everything already on the device with a
// margin of 4 GiB, and under a memory cap.
bool device_room(wavemoth_plan P, int64_t need) {
  size_t fr = 0, tot = 0;
  if (cudaMemGetInfo(&fr, &tot) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (int64_t)fr > need + (4LL << 30) &&
         !(g_device_cap > 0 && P->img->arena.bytes + P->arena.bytes + need > g_device_cap);
}

void free_host_direct(wm::HostProgram &G) {
  G.direct_ab.clear(); G.direct_ab.shrink_to_fit();
  G.direct_scale.clear(); G.direct_scale.shrink_to_fit();
  G.direct_tile_seeds.clear(); G.direct_tile_seeds.shrink_to_fit();
}

// Fills the plan's FP64 tables from its group columns.  FP64 images do not keep
// those: they pass through the plan's q buffer, in as many parts as that needs
// (allocating and freeing room for them took 0.7 of the 2.3 ms of a plan at nside
// 32); a shard, which has no q buffer, allocates.
int setup_direct(wavemoth_plan P) {
  auto &G = P->img->prog;
  const int64_t n = G.ngcols;
  if (!n) return 0;
  // the uploads went through the default stream, which the plan's does not wait for
  int rc = cuda_check(cudaStreamSynchronize(0), "image upload");
  wm::DevGCol *gcols = P->d_gcols, *own = nullptr;
  int64_t part = n;
  if (!gcols && P->nparts == 1) {
    gcols = reinterpret_cast<wm::DevGCol *>(P->d_q);
    const int64_t q_bytes = 2LL * (P->mmax + 1) * P->ni * P->nvecs * (int64_t)sizeof(double);
    part = std::min<int64_t>(n, q_bytes / (int64_t)sizeof(wm::DevGCol));
  } else if (!gcols) {
    rc = rc ? rc : cuda_check(cudaMalloc(&own, n * sizeof(wm::DevGCol)), "group columns");
    gcols = own;
  }
  if (!rc)
    rc = cuda_check(cudaMemsetAsync(P->d_direct_seeds, 0, std::max<int64_t>(G.direct_seeds, 1) * sizeof(double2),
                                    P->stream), "segment seeds");
  for (int64_t first = 0; first < n && !rc; first += part) {
    const int64_t count = std::min(part, n - first);
    if (!P->d_gcols)
      rc = cuda_check(cudaMemcpyAsync(gcols, G.gcols.data() + first, count * sizeof(wm::DevGCol),
                                      cudaMemcpyHostToDevice, P->stream), "group columns");
    if (!rc)
      rc = cuda_check(wm::launch_direct_setup(direct_params(P), gcols, first, count, P->d_f64, P->d_direct_cols,
                                              P->d_direct_inj, P->d_direct_seeds, P->stream), "column setup launch");
  }
  if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "column setup");
  cudaFree(own);
  return rc;
}

// The FP64 tables of a split image, at most 8 GiB (an nside 1024 plan's are 5)
// and where they fit; without them the plan keeps to the split GEMMs.
int provide_direct(wavemoth_plan P) {
  DeviceImage &I = *P->img;
  auto &G = I.prog;
  if (!I.direct) {
    const int64_t need = G.direct_seeds * (int64_t)sizeof(double2) +
                         G.ngcols * (int64_t)(sizeof(wm::DevDirectCol) + wm::kDirectInj * sizeof(double)) +
                         (int64_t)(G.direct_ab.size() + G.direct_scale.size()) * (int64_t)sizeof(double) + (64LL << 20);
    if (need > (8LL << 30) || !device_room(P, need)) return 0;
    DeviceArena A;
    A.base = I.arena.bytes + P->arena.bytes;
    ImageRefs R = I;
    if (build_direct(R, G, A)) {
      cudaGetLastError();  // another process took the memory
      return 0;
    }
    static_cast<ImageRefs &>(*P) = R;
    if (int rc = setup_direct(P)) return rc;
    static_cast<ImageRefs &>(I) = R;
    I.arena.adopt(A);
    free_host_direct(G);
  }
  static_cast<ImageRefs &>(*P) = I;
  return 0;
}

// The sliced residual P of a split image, where it fits; without it the GEMM
// kernels generate P at every call.
int provide_slices(wavemoth_plan P) {
  DeviceImage &I = *P->img;
  const auto &G = I.prog;
  if ((P->flags & WAVEMOTH_SPLIT_GENERATE) || G.stream_res_blocks <= 0) return 0;
  if (!I.d_res_a) {
    const int64_t need = G.stream_res_blocks * (int64_t)wm::kSplitBlock;
    if (!device_room(P, need)) return 0;
    DeviceArena A;
    A.base = I.arena.bytes + P->arena.bytes;
    if (A.alloc(&P->d_res_a, (size_t)need, "sliced residual P")) {
      cudaGetLastError();
      return 0;
    }
    const wm::SplitParams sp = split_params(P);
    int rc = cuda_check(wm::launch_residual_slices(sp, stream_launch(P, wm::kStreamResA2M),
                                                   stream_launch(P, wm::kStreamResM2A), P->stream),
                        "residual slice launch");
    if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "residual slices");
    if (rc) {
      P->d_res_a = nullptr;
      return rc;
    }
    I.d_res_a = P->d_res_a;
    I.res_a_bytes = need;
    I.arena.adopt(A);
  }
  P->d_res_a = I.d_res_a;
  P->res_a_bytes = I.res_a_bytes;
  return 0;
}

// Makes a split image hold what this plan's residual products read and earlier
// plans did not.  An nside 1024 image then has tens of GB of sliced P only if a
// plan of many maps reads it, and 5 GB of FP64 tables only if one of few does.
int provide_residual(wavemoth_plan P) {
  if (!P->split) return 0;
  if (prefers_direct(P))
    if (int rc = provide_direct(P)) return rc;
  return use_direct(P) ? 0 : provide_slices(P);
}

// Plan-time kernels of a new image, run through its first plan: ring
// tables, FP64 tables, recurrence seeds, split scales and level slices.
int init_image(wavemoth_plan P) {
  auto &G = P->img->prog;
  int rc = cuda_check(cudaStreamSynchronize(0), "image upload");  // as in setup_direct
  if (!rc) {
    wm::RingParams rp = ring_params(P);
    rc = cuda_check(wm::launch_ring_setup(rp, P->d_twiddles, P->max_bluestein ? P->d_filters : nullptr,
                                          P->d_ring_aux, P->d_phases, P->stream), "ring setup launch");
    if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "ring setup");
  }
  if (!rc && !P->split) rc = setup_direct(P);
  if (!rc && P->split && G.nseeds > 0) {
    wm::FastParams fp = fast_params(P);
    fp.seeds_out = P->d_seeds;
    rc = cuda_check(wm::launch_seeds(fp, P->stream), "seed kernel launch");
    if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "seed kernel");
  }
  if (!rc && P->split && !G.gcols.empty()) {
    // per-column and per-row maxima of P (scratch freed after use)
    unsigned long long *colmax = nullptr, *rowmax = nullptr;
    const size_t nc = G.gcols.size(), nr = (size_t)std::max<int64_t>(G.split_rows, 1);
    rc = cuda_check(cudaMalloc(&colmax, nc * sizeof(unsigned long long)), "scale scratch");
    if (!rc) rc = cuda_check(cudaMalloc(&rowmax, nr * sizeof(unsigned long long)), "scale scratch");
    if (!rc) rc = cuda_check(cudaMemsetAsync(rowmax, 0, nr * sizeof(unsigned long long), P->stream), "scale scratch");
    if (!rc) {
      wm::SplitParams sp = split_params(P);
      sp.colmax = colmax;
      sp.rowmax = rowmax;
      rc = cuda_check(wm::launch_split_scales(sp, P->stream), "split scale launch");
      if (!rc) rc = cuda_check(wm::launch_level_slices(sp, P->stream), "level slice launch");
      if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "split scales");
    }
    cudaFree(colmax);
    cudaFree(rowmax);
  }
  if (!rc) {
    // host-side tables that executes no longer need
    G.dblocks.clear(); G.dblocks.shrink_to_fit();
    G.strips.clear(); G.strips.shrink_to_fit();
    G.pairs.clear(); G.pairs.shrink_to_fit();
    G.f64.clear(); G.f64.shrink_to_fit();
    G.i32.clear(); G.i32.shrink_to_fit();
    G.gcols.clear(); G.gcols.shrink_to_fit();
    if (!P->split) free_host_direct(G);
  }
  return rc;
}

// Dense-recurrence plans: the first stored row of every (m, parity, ring)
// column (device ylmgen scan), the program, and after the image upload the
// stored seed values (device ylmgen fill).  eps as the reference's GPU
// precompute (wavemoth/cuda/sht.py:57, epsilon_legendre = 1e-30).
constexpr double kDenseEps = 1e-30;

struct DenseTemp {
  double *thetas = nullptr;
  int32_t *kstart = nullptr;
  ~DenseTemp() {
    cudaFree(thetas);
    cudaFree(kstart);
  }
};

int dense_scan(int nside, int lmax, int mmax, DenseTemp &T, std::vector<int32_t> &kstart) {
  const int ni = 2 * nside;
  std::vector<double> th = wm::ring_pair_z(nside);
  for (double &v : th) v = acos(v);
  kstart.assign(2 * (size_t)(mmax + 1) * ni, 0);
  int rc = cuda_check(cudaMalloc(&T.thetas, th.size() * sizeof(double)), "dense scan buffers");
  rc = rc ? rc : cuda_check(cudaMalloc(&T.kstart, kstart.size() * sizeof(int32_t)), "dense scan buffers");
  rc = rc ? rc : cuda_check(cudaMemcpy(T.thetas, th.data(), th.size() * sizeof(double), cudaMemcpyHostToDevice),
                            "dense scan upload");
  rc = rc ? rc : cuda_check(wm::launch_dense_scan(lmax, mmax, T.thetas, ni, kDenseEps, T.kstart, 0), "dense scan");
  rc = rc ? rc : cuda_check(cudaMemcpy(kstart.data(), T.kstart, kstart.size() * sizeof(int32_t),
                                       cudaMemcpyDeviceToHost), "dense scan download");
  return rc;
}

// Per ring pair, 1 + the largest m whose column (either parity) has a row
// above the scan's threshold (kstart < nk): the synthesis gather's m limit.
std::vector<int32_t> ring_m_limits(int nside, int lmax, int mmax, const std::vector<int32_t> &kstart) {
  const int64_t ni = 2LL * nside;
  std::vector<int32_t> mend((size_t)ni, 0);
  for (int m = 0; m <= mmax; ++m)
    for (int p = 0; p < 2; ++p) {
      const int32_t nk = lmax - m - p >= 0 ? (lmax - m - p) / 2 + 1 : 0;
      const int32_t *ks = kstart.data() + (size_t)(2 * m + p) * ni;
      for (int64_t r = 0; r < ni; ++r)
        if (ks[r] < nk) mend[(size_t)r] = m + 1;
    }
  return mend;
}

int dense_fill(const DeviceImage &I, DenseTemp &T, const std::vector<wm::DevDenseFill> &fill) {
  wm::DevDenseFill *d_fill = nullptr;
  int rc = cuda_check(cudaMalloc(&d_fill, std::max<size_t>(fill.size(), 1) * sizeof(wm::DevDenseFill)), "dense fill");
  rc = rc ? rc : cuda_check(cudaMemcpy(d_fill, fill.data(), fill.size() * sizeof(wm::DevDenseFill),
                                       cudaMemcpyHostToDevice), "dense fill upload");
  rc = rc ? rc : cuda_check(wm::launch_dense_fill(I.prog.lmax, I.prog.mmax, T.thetas, 2 * I.prog.nside, kDenseEps,
                                                  T.kstart, d_fill, I.d_f64, 0), "dense fill");
  rc = rc ? rc : cuda_check(cudaDeviceSynchronize(), "dense fill");
  cudaFree(d_fill);
  return rc;
}

// Everything wavemoth_legendre_alm2map_noalloc needs from the driver, done
// while allocating is allowed: the device address of its static scratch
// array (resolving it loads the module that holds the array, which is when
// the array's memory is taken) and the module of the kernel it launches.
int prepare_noalloc() {
  void *addr = nullptr;
  size_t bytes = 0;
  std::string err;
  if (wm::noalloc_scratch(&addr, &bytes, err)) return set_error(WAVEMOTH_ERR_CUDA, err);
  return cuda_check(wm::legendre_preload(), "loading the Legendre kernels");
}

// Contiguous split of items 0..n-1 with the given costs into nparts ranges
// of about equal cost: bounds[k] .. bounds[k + 1] (bounds[0] = 0,
// bounds[nparts] = n); every range non-empty when n >= nparts.
std::vector<int64_t> balanced_ranges(const std::vector<double> &cost, int nparts) {
  const int64_t n = (int64_t)cost.size();
  double total = 0.0;
  for (double c : cost) total += c;
  std::vector<int64_t> b(nparts + 1, n);
  b[0] = 0;
  double acc = 0.0;
  int64_t i = 0;
  for (int k = 1; k < nparts; ++k) {
    const double target = total * k / nparts;
    while (i < n && (acc + 0.5 * cost[i] < target || i < b[k - 1] + 1)) acc += cost[i++];
    b[k] = std::min(i, n - (nparts - k));  // leave at least one item per later part
    while (i < b[k]) acc += cost[i++];
    while (i > b[k]) acc -= cost[--i];
  }
  return b;
}

wavemoth_plan make_plan(bool analysis, int Nside, int lmax, int mmax, int nmaps, double *input,
                        double *output, int ordering, unsigned flags, const char *resource_filename,
                        int nparts = 1, int part = 0) {
  if (nparts < 1 || part < 0 || part >= nparts || (nparts > 1 && !(flags & WAVEMOTH_DEVICE_POINTERS))) {
    set_error(WAVEMOTH_ERR_ARG, "invalid shard (need 0 <= part < nparts; shards take device pointers)");
    return nullptr;
  }
  if (nmaps <= 0 || lmax < 0 || mmax != lmax || ordering != WAVEMOTH_MMAJOR) {
    set_error(WAVEMOTH_ERR_ARG, "invalid plan arguments (need nmaps > 0, mmax == lmax >= 0, "
                                "ordering WAVEMOTH_MMAJOR)");
    return nullptr;
  }
  std::string path;
  const bool dense = (flags & WAVEMOTH_DENSE) != 0;
  if (dense) {
    if (Nside <= 0) {
      set_error(WAVEMOTH_ERR_ARG, "a dense-recurrence plan needs Nside > 0");
      return nullptr;
    }
    path = "<dense recurrence, nside " + std::to_string(Nside) + ">";
  } else if (resource_filename) {
    path = resource_filename;
  } else {
    if (Nside <= 0 || g_resource_dir.empty()) {
      set_error(WAVEMOTH_ERR_ARG, "no resource file given and wavemoth_configure not called");
      return nullptr;
    }
    path = g_resource_dir + "/rev1/" + std::to_string(Nside) + ".dat";
  }
  struct stat st {};
  if (!dense && stat(path.c_str(), &st) != 0) {
    set_error(WAVEMOTH_ERR_RESOURCE, "cannot open resource file " + path);
    return nullptr;
  }
  const unsigned image_flags = flags & (WAVEMOTH_PRECISION_SPLIT | WAVEMOTH_SPLIT_GENERATE | WAVEMOTH_DENSE);
  const ImageKey key{path, (int64_t)st.st_size, (int64_t)st.st_mtime, lmax, mmax, image_flags, nparts, part};
  std::lock_guard<std::mutex> lock(g_image_mutex);
  std::shared_ptr<DeviceImage> img = g_images.count(key) ? g_images[key].lock() : nullptr;
  const bool fresh = !img;
  std::string err;
  if (fresh) {
    img = std::make_shared<DeviceImage>();
    DenseTemp dtemp;
    std::vector<wm::DevDenseFill> dfill;
    std::vector<int32_t> kstart;  // first active row of every (m, parity, ring) column
    if (dense) {
      if (dense_scan(Nside, lmax, mmax, dtemp, kstart)) return nullptr;
      if (!wm::build_dense_program(Nside, lmax, mmax, kstart, img->prog, dfill, err)) {
        set_error(WAVEMOTH_ERR_ARG, err);
        return nullptr;
      }
    } else {
      std::vector<char> file;
      if (!read_file(path, file, err)) {
        set_error(WAVEMOTH_ERR_RESOURCE, err);
        return nullptr;
      }
      if (!wm::compile_resource(file.data(), file.size(), Nside, lmax, mmax, img->prog, err)) {
        set_error(WAVEMOTH_ERR_RESOURCE, path + ": " + err);
        return nullptr;
      }
    }
    if (nparts > 1) {
      // this part's m range, balanced by the matrices' estimated work
      std::vector<double> cost(mmax + 1, 0.0);
      for (const auto &M : img->prog.mats) cost[M.m] += M.cost + 1.0;
      img->m_bounds = balanced_ranges(cost, nparts);
      img->prog.shard_m0 = (int32_t)img->m_bounds[part];
      img->prog.shard_m1 = (int32_t)img->m_bounds[part + 1];
    }
    if (!wm::build_fast_path(img->prog, (image_flags & WAVEMOTH_PRECISION_SPLIT) != 0, err)) {
      set_error(WAVEMOTH_ERR_RESOURCE, path + ": " + err);
      return nullptr;
    }
    if (nparts == 1) {
      if (kstart.empty() && dense_scan(img->prog.nside, lmax, mmax, dtemp, kstart)) return nullptr;
      img->prog.ring_mend = ring_m_limits(img->prog.nside, lmax, mmax, kstart);
    }
    if (build_image(*img, img->prog.nside, mmax, image_flags)) return nullptr;
    if (dense && dense_fill(*img, dtemp, dfill)) return nullptr;
  } else if (Nside > 0 && img->prog.nside != Nside) {
    set_error(WAVEMOTH_ERR_RESOURCE, path + ": file is for another Nside");
    return nullptr;
  }
  auto *P = new _wavemoth_plan();
  P->img = img;
  if (!dense) P->resource_path = path;
  auto &G = img->prog;
  P->nside = G.nside;
  P->lmax = lmax;
  P->mmax = mmax;
  P->nmaps = nmaps;
  P->nvecs = 2 * nmaps;
  P->ni = 2 * P->nside;
  P->npix = 12LL * P->nside * P->nside;
  P->nalm = (int64_t)(lmax + 1) * (lmax + 2) / 2;
  P->flags = flags;
  P->analysis = analysis;
  P->host_in = input;
  P->host_out = output;

  int dev = 0;
  if (cuda_check(cudaGetDevice(&dev), "cudaGetDevice") ||
      cuda_check(cudaDeviceGetAttribute(&P->sm_count, cudaDevAttrMultiProcessorCount, dev),
                 "cudaDeviceGetAttribute")) {
    delete P;
    return nullptr;
  }
  const int nmats = (int)G.mats.size();
  P->grid = std::max(1, std::min(nmats, 2 * P->sm_count));
  P->slot_stride = 2 * (int64_t)std::max<int32_t>(G.max_rows, 1) * P->nvecs;
  int rc = 0;
  DeviceArena &A = P->arena;
  A.base = img->arena.bytes;
  rc = rc ? rc : A.alloc(&P->d_xbuf, (size_t)std::max<int64_t>(G.xrows, 1) * P->nvecs, "X buffer");
  P->nparts = nparts;
  P->part = part;
  {
    RingTable RT = ring_table(P->nside, nmaps, mmax);
    if (!rc && RT.max_cta_cplx > wm::kRingBufferCplx)
      rc = set_error(WAVEMOTH_ERR_ARG, "ring transforms longer than 8192 points (nside > 2048) are not supported");
    if (nparts > 1) {
      // this part's ring pairs, a contiguous range balanced by pixels
      std::vector<double> cost(P->ni);
      for (int r = 0; r < P->ni; ++r) cost[r] = (double)RT.rings[r].n * (r ? 2.0 : 1.0);
      P->ring_bounds = balanced_ranges(cost, nparts);
      P->m_bounds = img->m_bounds;
      const int64_t r0 = P->ring_bounds[part], r1 = P->ring_bounds[part + 1];
      std::vector<wm::DevRingTask> mine;
      for (const auto &t : RT.tasks)
        if (t.ring >= r0 && t.ring < r1) mine.push_back(t);
      RT.tasks.swap(mine);
      // exchange table: per m, the offset of its rows in the ring-side
      // exchange buffer [source part][ring of this part][m of that part][parity]
      // and their stride from one ring to the next (doubles)
      std::vector<int64_t> tab(2 * (size_t)(mmax + 1));
      int64_t seg = 0;
      for (int s = 0; s < nparts; ++s) {
        const int64_t m0 = P->m_bounds[s], cnt = P->m_bounds[s + 1] - m0;
        for (int64_t m = m0; m < m0 + cnt; ++m) {
          tab[2 * m] = seg + (m - m0) * 2 * P->nvecs;
          tab[2 * m + 1] = cnt * 2 * P->nvecs;
        }
        seg += (r1 - r0) * cnt * 2 * P->nvecs;
      }
      rc = rc ? rc : upload(A, &P->d_shard_tab, tab, "shard exchange table");
    }
    P->ring_ntasks = (int32_t)RT.tasks.size();
    P->ring_smem = RT.smem;
    P->ring_threads = RT.threads;
    P->ring_short = RT.short_rings;
    rc = rc ? rc : upload(A, &P->d_ring_tasks, RT.tasks, "ring work list");
  }
  if (img->split) {
    rc = rc ? rc : A.alloc(&P->d_vec_scale, (size_t)std::max<size_t>(G.groups.size() + G.roots.size(), 1) *
                                                wm::kSplitN, "vector scales");
    rc = rc ? rc : A.alloc(&P->d_planes, (size_t)std::max<int64_t>(G.split_chunks, 1) * wm::kSplitPlane,
                           "operand slices");
  }
  rc = rc ? rc : A.alloc(&P->d_status, 1, "status word");
  rc = rc ? rc : A.alloc(&P->d_counter, 1, "counter");
  // (a shard's q buffers are the caller's exchange buffers)
  rc = rc ? rc : A.alloc(&P->d_q, nparts > 1 ? 1 : (size_t)2 * (mmax + 1) * P->ni * P->nvecs, "q buffer");
  rc = rc ? rc : A.alloc(&P->d_scratch, (size_t)P->grid * P->slot_stride, "butterfly scratch");
  if (!(flags & WAVEMOTH_DEVICE_POINTERS)) {
    rc = rc ? rc : A.alloc(&P->d_alm, (size_t)P->nalm * P->nvecs, "alm buffer");
    rc = rc ? rc : A.alloc(&P->d_map, (size_t)P->npix * nmaps, "map buffer");
  }
  static_cast<ImageRefs &>(*P) = static_cast<const ImageRefs &>(*img);
  rc = rc ? rc : cuda_check(cudaStreamCreateWithFlags(&P->stream, cudaStreamNonBlocking),
                            "cudaStreamCreate");
  if (!rc) rc = cuda_check(cudaMemsetAsync(P->d_status, 0, sizeof(int32_t), P->stream), "status reset");
  if (!rc && fresh) rc = init_image(P);
  if (!rc) rc = provide_residual(P);
  A.base = img->arena.bytes;
  if (!rc) rc = cuda_check(cudaStreamSynchronize(P->stream), "plan setup");
  if (!rc) rc = prepare_noalloc();
  if (rc) {
    delete P;
    return nullptr;
  }
  if (fresh) g_images[key] = img;
  return P;
}

wm::LegendreParams legendre_params(wavemoth_plan P) {
  wm::LegendreParams p{};
  p.mats = P->d_mats;
  p.dblocks = P->d_dblocks;
  p.strips = P->d_strips;
  p.levels = P->d_levels;
  p.pairs = P->d_pairs;
  p.f64 = P->d_f64;
  p.i32 = P->d_i32;
  p.order = P->d_order;
  p.nmats = (int32_t)P->img->prog.mats.size();
  p.lmax = P->lmax;
  p.nvecs = P->nvecs;
  p.ni = P->ni;
  p.q_mstride = P->nvecs;
  p.q_rstride = 2LL * shard_mcount(P) * P->nvecs;
  p.scratch = P->d_scratch;
  p.slot_stride = P->slot_stride;
  p.counter = P->d_counter;
  return p;
}

}  // namespace

namespace wm {

int set_last_error(int code, const std::string &msg) { return set_error(code, msg); }

// Legendre kernel parameters of a plan (program tables, sizes, grid) without
// any buffers bound; used by entry points that bring their own buffers.
bool plan_legendre_params(wavemoth_plan plan, LegendreParams &p, int &grid, std::string &err) {
  if (!plan) {
    err = "NULL plan";
    return false;
  }
  p = legendre_params(plan);
  grid = plan->grid;
  return true;
}

}  // namespace wm

namespace {

wm::RingParams ring_params(wavemoth_plan P) {
  wm::RingParams r{};
  r.rings = P->d_rings;
  r.ni = P->ni;
  r.nside = P->nside;
  r.mmax = P->mmax;
  r.nmaps = P->nmaps;
  r.nvecs = P->nvecs;
  r.scale = 4.0 * 3.14159265358979323846 / (double)P->npix;
  r.map_scale = 1.0;
  r.ring_weights = P->d_ring_weights;
  r.phase_shifts = P->phase_shifts;
  r.twiddles = reinterpret_cast<const double2 *>(P->d_twiddles);
  r.twlen = P->twlen;
  r.filters = P->d_filters;
  r.aux = reinterpret_cast<const double2 *>(P->d_ring_aux);
  r.max_bluestein_m = P->max_bluestein;
  r.tasks = P->d_ring_tasks;
  r.ntasks = P->ring_ntasks;
  r.smem = P->ring_smem;
  r.threads = P->ring_threads;
  r.short_rings = P->ring_short;
  r.nphase_hi = P->nphase_hi;
  r.phases = P->d_phases;
  return r;
}

// kinds: 0 Legendre alm2map, 1 Legendre map2alm, 2 ring synthesis, 3 ring analysis
int span_begin(wavemoth_plan P, int kind, cudaStream_t st) {
  if (!P->timing) return -1;
  _wavemoth_plan::Span s{kind, nullptr, nullptr};
  if (cudaEventCreate(&s.a) != cudaSuccess || cudaEventCreate(&s.b) != cudaSuccess) return -1;
  cudaEventRecord(s.a, st);
  P->spans.push_back(s);
  return (int)P->spans.size() - 1;
}

void span_end(wavemoth_plan P, int idx, cudaStream_t st) {
  if (idx >= 0) cudaEventRecord(P->spans[idx].b, st);
}

// SMs the plan's persistent Legendre kernels may occupy (the batch
// scheduler's cap, else all)
int plan_sms(wavemoth_plan P) { return P->grid_cap > 0 ? std::min(P->grid_cap, P->sm_count) : P->sm_count; }

// Split-precision residual products, kSplitN vectors per pass: operand
// slices of the pass, then the tensor-core GEMM of every group tile.
// Launch description of streamed split GEMM k (wm::kStream*).
wm::StreamLaunch stream_launch(wavemoth_plan P, int k) {
  wm::StreamLaunch L{};
  L.tiles = P->d_stream_tiles[k];
  L.rows = P->d_stream_rows[k];
  L.sidx = P->d_stream_sidx[k];
  L.ntiles = P->nstream[k];
  if (k == wm::kStreamResA2M || k == wm::kStreamResM2A) {
    L.scales = k == wm::kStreamResA2M ? P->d_col_scale : P->d_row_scale;
    L.a = P->d_res_a;
    L.a_mn = k == wm::kStreamResM2A;
  } else {
    L.scales = P->d_level_rs;
    L.a = P->d_level_a;
    L.a_mn = 0;
  }
  return L;
}

int run_split(wavemoth_plan P, bool alm2map, const double *alm_in, double *alm_out, const double *q_in,
              double *q_out, cudaStream_t st) {
  const auto &G = P->img->prog;
  if (G.groups.empty()) return 0;
  wm::SplitParams s = split_params(P);
  s.alm_in = alm_in;
  s.alm_out = alm_out;
  s.q_in = q_in;
  s.q = q_out;
  const int nt = alm2map ? s.ntiles_a : s.ntiles_b;
  const int nl = alm2map ? s.ntiles_la : s.ntiles_lm;
  const int gop = std::min((int)G.groups.size(), 8 * P->sm_count);
  const int gop_l = std::min(std::max(s.nroots, 1), 8 * P->sm_count);
  for (int v0 = 0; v0 < P->nvecs; v0 += wm::kSplitN) {
    s.v0 = v0;
    int rc = 0;
    // alm2map: residual (alm -> X, q) then levels (X -> q); map2alm reversed
    // rows that no tile of launch k writes read as zero
    auto zero_rows = [&](int k) {
      if (rc || !P->nsplit_zero[k]) return;
      rc = cuda_check(wm::launch_zero_rows(s, P->d_split_zero[k], P->nsplit_zero[k], st), "zero rows launch");
      P->kernel_launches++;
    };
    auto residual = [&]() {
      rc = cuda_check(wm::launch_split(alm2map ? 0 : 2, s, gop, st), "operand slice launch");
      P->kernel_launches++;
      zero_rows(alm2map ? wm::kStreamResA2M : wm::kStreamResM2A);
      if (rc || !nt) return;
      if (P->d_res_a) {
        const wm::StreamLaunch L = stream_launch(P, alm2map ? wm::kStreamResA2M : wm::kStreamResM2A);
        rc = cuda_check(wm::launch_stream(s, L, std::min(L.ntiles, plan_sms(P)), st), "split GEMM launch");
      } else {
        rc = cuda_check(wm::launch_split(alm2map ? 1 : 3, s, std::min(nt, plan_sms(P)), st), "split GEMM launch");
      }
      P->kernel_launches++;
    };
    auto levels = [&]() {
      zero_rows(alm2map ? wm::kStreamLevelA2M : wm::kStreamLevelM2A);
      if (rc || !nl) return;
      rc = cuda_check(wm::launch_split(alm2map ? 4 : 6, s, gop_l, st), "level operand slice launch");
      P->kernel_launches++;
      if (!rc) {
        const wm::StreamLaunch L = stream_launch(P, alm2map ? wm::kStreamLevelA2M : wm::kStreamLevelM2A);
        rc = cuda_check(wm::launch_stream(s, L, std::min(L.ntiles, plan_sms(P)), st), "level GEMM launch");
        P->kernel_launches++;
      }
    };
    if (alm2map) {
      residual();
      if (!rc) levels();
    } else {
      levels();
      if (!rc) residual();
    }
    if (rc) return rc;
  }
  return 0;
}

// What map2alm does with the alm it computes: writes it, adds it, or writes it
// as the gradient of a real map (rows of m > 0 twice, Im a_l0 zero).
enum class AlmOut { kWrite, kAdd, kBackward };

// FP64 path: residual products, and the interpolation levels of depth-1
// matrices after (alm2map) or before them (map2alm).
int run_direct(wavemoth_plan P, bool alm2map, const double *alm_in, double *alm_out, const double *q_in,
               double *q_out, cudaStream_t st, AlmOut how) {
  const auto &G = P->img->prog;
  const int nr = (int)G.roots.size(), cap = P->grid_cap > 0 ? 4 * plan_sms(P) : 0;
  int rc = 0;
  auto levels = [&]() {
    if (rc || !nr) return;
    wm::FastParams f = fast_params(P);
    f.q_in = q_in;
    f.q = q_out;
    rc = cuda_check(wm::launch_level(alm2map, f, cap, st), "level launch");
    P->kernel_launches++;
  };
  wm::DirectParams d = direct_params(P);
  d.alm_in = alm_in;
  d.alm_out = alm_out;
  d.q_in = q_in;
  d.q = q_out;
  d.accumulate = how == AlmOut::kAdd;
  d.backward = how == AlmOut::kBackward;
  if (alm2map) {
    d.aligned = (((uintptr_t)q_out | (uintptr_t)alm_in) & 15) == 0;
    rc = cuda_check(wm::launch_direct_a2m(d, P->d_direct_a, P->ndirect_a, plan_sms(P), cap, st),
                    "alm2map residual launch");
    P->kernel_launches += P->ndirect_a[0] > 0;
    levels();
  } else {
    levels();
    if (!rc) rc = cuda_check(wm::launch_direct_m2a(d, cap, st), "map2alm residual launch");
    P->kernel_launches += d.ntiles_b > 0;
  }
  return rc;
}

int run_legendre(wavemoth_plan P, bool alm2map, const double *alm_in, double *alm_out,
                 const double *q_in, double *q_out, cudaStream_t st, AlmOut how = AlmOut::kWrite) {
  const auto &G = P->img->prog;
  int sp = span_begin(P, alm2map ? 0 : 1, st);
  int rc = 0;
  if (!use_direct(P)) {
    rc = run_split(P, alm2map, alm_in, alm_out, q_in, q_out, st);
  } else {
    rc = run_direct(P, alm2map, alm_in, alm_out, q_in, q_out, st, how);
  }
  if (!rc && P->nslow > 0) {
    wm::LegendreParams p = legendre_params(P);
    p.order = P->d_order_slow;
    p.nmats = P->nslow;
    p.alm_in = alm_in;
    p.alm_out = alm_out;
    p.q_in = q_in;
    p.q_out = q_out;
    rc = cuda_check(cudaMemsetAsync(P->d_counter, 0, sizeof(int32_t), st), "counter reset");
    if (!rc)
      rc = cuda_check(wm::launch_legendre(alm2map, p, std::min(P->grid, std::max(1, (int)P->nslow)), st),
                      "Legendre kernel launch");
    P->kernel_launches++;
  }
  span_end(P, sp, st);
  return rc;
}

// Whether the plan's map2alm can do more than write the alm (AlmOut): every
// matrix on the FP64 units.
bool weighs_alm(wavemoth_plan P) { return use_direct(P) && P->nslow == 0; }

// scale multiplies the maps (1 for alm2map; 4 pi / npix for the adjoint of
// map2alm); sub, if given, is what they are subtracted from
int run_alm2map(wavemoth_plan P, const double *alm, double *map, cudaStream_t st, double scale = 1.0,
                const double *sub = nullptr) {
  if (int rc = run_legendre(P, true, alm, nullptr, nullptr, P->d_q, st)) return rc;
  wm::RingParams r = ring_params(P);
  r.q = P->d_q;
  // q was just written by this plan's Legendre step: its rows above each
  // ring's m limit hold at most 1e-30 |a| (Legendre values below the plan
  // writer's inclusion threshold), and the gather stops there
  r.ring_mend = P->d_ring_mend;
  r.map = map;
  r.map_sub = sub;
  r.map_scale = scale;
  int sp = span_begin(P, 2, st);
  int rc = cuda_check(wm::launch_ring_synthesis(r, st), "ring synthesis launch");
  P->kernel_launches += r.ntasks > 0;
  span_end(P, sp, st);
  return rc;
}

// map2alm, or (adjoint) (npix / 4 pi) times it without the ring weights, the
// adjoint of alm2map
int run_map2alm(wavemoth_plan P, const double *map, double *alm, cudaStream_t st, bool adjoint = false,
                AlmOut how = AlmOut::kWrite) {
  wm::RingParams r = ring_params(P);
  if (adjoint) {
    r.scale = 1.0;
    r.ring_weights = nullptr;
  }
  r.map_in = map;
  r.q_out = P->d_q;
  // q~ is consumed by this plan's Legendre step, which weighs the rows above
  // each ring's m limit by Legendre values below 1e-30: written as zeros
  r.ring_mend = P->d_ring_mend;
  int sp = span_begin(P, 3, st);
  int rc0 = cuda_check(wm::launch_ring_analysis(r, st), "ring analysis launch");
  P->kernel_launches += r.ntasks > 0;
  span_end(P, sp, st);
  if (rc0) return rc0;
  return run_legendre(P, false, nullptr, alm, P->d_q, nullptr, st, how);
}

// Reads (and clears) the device status word; the stream must be idle.
int device_status(wavemoth_plan P) {
  int32_t st = 0;
  int rc = cuda_check(cudaMemcpy(&st, P->d_status, sizeof(st), cudaMemcpyDeviceToHost), "status read");
  if (rc) return rc;
  if (st == 0) return 0;
  cudaMemset(P->d_status, 0, sizeof(st));
  return set_error(WAVEMOTH_ERR_DEVICE, st == wm::kStatusTimeout ? "a kernel's bounded wait expired"
                                                                 : "a kernel reported a bad program table");
}

int finish(wavemoth_plan P, int rc) {
  P->status = rc;
  return rc;
}

// Whole transforms and hooks on their q need the plan's own q buffer, which a
// shard does not have (its q buffers are the caller's).
int whole_plan_check(wavemoth_plan P, const void *a, const void *b) {
  if (!P || !a || !b) return set_error(WAVEMOTH_ERR_ARG, "NULL plan or buffer");
  if (P->nparts > 1)
    return set_error(WAVEMOTH_ERR_ARG, "a shard of a plan runs through the wavemoth_shard_ calls only");
  return 0;
}

// The plan's transform on its bound buffers (input -> output), or with
// adjoint its adjoint (output -> input): for an alm2map plan
// A^T f = (npix / 4 pi) map2alm(f), for a map2alm plan (4 pi / npix)
// alm2map(a) times the ring weights, both with respect to the real inner product on maps and
// <a, b> = sum_lm c_m Re(a_lm conj b_lm) (c_0 = 1, c_m = 2) on alm.
int host_execute(wavemoth_plan P, bool adjoint = false) {
  cudaStream_t st = P->stream;
  const bool devptr = (P->flags & WAVEMOTH_DEVICE_POINTERS) != 0;
  const size_t alm_bytes = (size_t)P->nalm * P->nvecs * sizeof(double);
  const size_t map_bytes = (size_t)P->npix * P->nmaps * sizeof(double);
  if (!P->host_in || !P->host_out)
    return set_error(WAVEMOTH_ERR_ARG, "plan has no bound input/output buffers");
  int rc = 0;
  const bool synthesis = P->analysis == adjoint;
  double *alm_host = P->analysis ? P->host_out : P->host_in;
  double *map_host = P->analysis ? P->host_in : P->host_out;
  if (synthesis) {
    const double *alm = devptr ? alm_host : P->d_alm;
    double *map = devptr ? map_host : P->d_map;
    if (!devptr)
      rc = cuda_check(cudaMemcpyAsync(P->d_alm, alm_host, alm_bytes, cudaMemcpyHostToDevice, st),
                      "alm upload");
    rc = rc ? rc : run_alm2map(P, alm, map, st, adjoint ? 4.0 * 3.14159265358979323846 / (double)P->npix : 1.0);
    if (adjoint && !rc && P->d_ring_weights)
      rc = cuda_check(wm::launch_ring_weights(P->d_rings, P->ni, P->d_ring_weights, P->nmaps, map, st),
                      "ring weights launch");
    if (!devptr && !rc)
      rc = cuda_check(cudaMemcpyAsync(map_host, P->d_map, map_bytes, cudaMemcpyDeviceToHost, st),
                      "map download");
  } else {
    const double *map = devptr ? map_host : P->d_map;
    double *alm = devptr ? alm_host : P->d_alm;
    if (!devptr)
      rc = cuda_check(cudaMemcpyAsync(P->d_map, map_host, map_bytes, cudaMemcpyHostToDevice, st),
                      "map upload");
    rc = rc ? rc : run_map2alm(P, map, alm, st, adjoint);
    if (!devptr && !rc)
      rc = cuda_check(cudaMemcpyAsync(alm_host, P->d_alm, alm_bytes, cudaMemcpyDeviceToHost, st),
                      "alm download");
  }
  if (!rc) rc = cuda_check(cudaStreamSynchronize(st), "execute");
  if (!rc) rc = device_status(P);
  return rc;
}

}  // namespace

namespace wm {

// Batch coalescing (batch.cpp): two device-pointer plans compute the same
// transform on their maps when they share the device image (file, lmax,
// mmax, precision) and the settings that change results or bound their waits.
bool plans_coalescible(wavemoth_plan a, wavemoth_plan b) {
  return a && b && a != b && a->img == b->img && a->flags == b->flags && a->lmax == b->lmax &&
         a->mmax == b->mmax && a->phase_shifts == b->phase_shifts && a->wait_limit == b->wait_limit &&
         !a->d_ring_weights && !b->d_ring_weights && a->nparts == 1 && b->nparts == 1 &&
         (a->flags & WAVEMOTH_DEVICE_POINTERS);
}

// A device-pointer plan of `nmaps` maps on the image of P (no new image).
wavemoth_plan plan_with_maps(wavemoth_plan P, int nmaps) {
  const bool dense = (P->flags & WAVEMOTH_DENSE) != 0;
  wavemoth_plan Q = make_plan(P->analysis, P->nside, P->lmax, P->mmax, nmaps, nullptr, nullptr, WAVEMOTH_MMAJOR,
                              P->flags | WAVEMOTH_DEVICE_POINTERS, dense ? nullptr : P->resource_path.c_str());
  if (Q) {
    Q->phase_shifts = P->phase_shifts;
    if (wavemoth_plan_set_wait_limit(Q, P->wait_limit)) {
      delete Q;
      return nullptr;
    }
  }
  return Q;
}

void plan_sizes(wavemoth_plan P, int64_t *nalm, int64_t *npix) {
  *nalm = P->nalm;
  *npix = P->npix;
}

}  // namespace wm

extern "C" {

const char *wavemoth_last_error(void) { return g_last_error.c_str(); }

void wavemoth_configure(char *resource_dir) { g_resource_dir = resource_dir ? resource_dir : ""; }

wavemoth_plan wavemoth_plan_to_healpix(int Nside, int lmax, int mmax, int nmaps, int nthreads,
                                       double *input, double *output, int ordering,
                                       unsigned flags, char *resource_filename) {
  (void)nthreads;
  return make_plan(false, Nside, lmax, mmax, nmaps, input, output, ordering, flags,
                   resource_filename);
}

wavemoth_plan wavemoth_plan_from_healpix(int Nside, int lmax, int mmax, int nmaps, int nthreads,
                                         double *input, double *output, int ordering,
                                         unsigned flags, char *resource_filename) {
  (void)nthreads;
  return make_plan(true, Nside, lmax, mmax, nmaps, input, output, ordering, flags,
                   resource_filename);
}

void wavemoth_destroy_plan(wavemoth_plan plan) {
  if (!plan) return;
  if (plan->stream) cudaStreamSynchronize(plan->stream);
  delete plan;
}

void wavemoth_execute(wavemoth_plan plan) {
  if (!plan) {
    set_error(WAVEMOTH_ERR_ARG, "NULL plan");
    return;
  }
  finish(plan, host_execute(plan));
}

void wavemoth_execute_adjoint(wavemoth_plan plan) {
  if (!plan) {
    set_error(WAVEMOTH_ERR_ARG, "NULL plan");
    return;
  }
  finish(plan, host_execute(plan, true));
}

int wavemoth_plan_status(wavemoth_plan plan) { return plan ? plan->status : WAVEMOTH_ERR_ARG; }

int wavemoth_plan_device_status(wavemoth_plan plan, void *stream) {
  if (!plan) return set_error(WAVEMOTH_ERR_ARG, "NULL plan");
  if (int rc = cuda_check(cudaStreamSynchronize((cudaStream_t)stream), "device status")) return rc;
  return finish(plan, device_status(plan));
}

int64_t wavemoth_get_legendre_flops(wavemoth_plan plan, int m, int odd) {
  if (!plan || m < 0 || m > plan->mmax || odd < 0 || odd > 1) return -1;
  return plan->img->prog.element_count[2 * m + odd] * 2 * 2;
}

int wavemoth_query_resourcefile(char *filename, int *out_Nside, int *out_lmax) {
  if (!filename) return -1;
  FILE *f = fopen(filename, "rb");
  if (!f) return -1;
  int64_t fields[3];
  size_t got = fread(fields, sizeof(fields), 1, f);
  fclose(f);
  if (got != 1) {
    set_error(WAVEMOTH_ERR_RESOURCE, std::string("could not read file header: ") + filename);
    return -1;
  }
  *out_lmax = (int)fields[0];
  *out_Nside = (int)fields[2];
  return 0;
}

int wavemoth_execute_alm2map_device(wavemoth_plan plan, const double *alm, double *map,
                                    void *stream) {
  if (int rc = whole_plan_check(plan, alm, map)) return rc;
  return finish(plan, run_alm2map(plan, alm, map, (cudaStream_t)stream));
}

int wavemoth_execute_map2alm_device(wavemoth_plan plan, const double *map, double *alm,
                                    void *stream) {
  if (int rc = whole_plan_check(plan, alm, map)) return rc;
  return finish(plan, run_map2alm(plan, map, alm, (cudaStream_t)stream));
}

wavemoth_plan wavemoth_plan_shard(int Nside, int lmax, int mmax, int nmaps, unsigned flags,
                                  char *resource_filename, int nparts, int part) {
  return make_plan(false, Nside, lmax, mmax, nmaps, nullptr, nullptr, WAVEMOTH_MMAJOR,
                   flags | WAVEMOTH_DEVICE_POINTERS, resource_filename, nparts, part);
}

int wavemoth_shard_layout(wavemoth_plan plan, int64_t *m_bounds, int64_t *ring_bounds) {
  if (!plan || plan->nparts < 2 || !m_bounds || !ring_bounds)
    return set_error(WAVEMOTH_ERR_ARG, "wavemoth_shard_layout: not a sharded plan");
  for (int k = 0; k <= plan->nparts; ++k) {
    m_bounds[k] = plan->m_bounds[k];
    ring_bounds[k] = plan->ring_bounds[k];
  }
  return 0;
}

}  // extern "C"

namespace {

int shard_check(wavemoth_plan P, const void *a, const void *b) {
  if (!P || P->nparts < 2 || !a || !b) return set_error(WAVEMOTH_ERR_ARG, "not a sharded plan, or a NULL buffer");
  return 0;
}

// The shard's q buffer (rows of its own m) addressed as a full q: the
// kernels index row (m, parity, ring) at (2m + parity) + 2 ring mcount.
template <class T>
T *q_origin(wavemoth_plan P, T *q) {
  return q - 2 * P->m_bounds[P->part] * P->nvecs;
}

// ring-side q of the shard's ring pairs r0..r1 addressed as a full q
template <class T>
T *ring_origin(wavemoth_plan P, T *q) {
  return q - P->ring_bounds[P->part] * 2 * ((int64_t)P->mmax + 1) * P->nvecs;
}

}  // namespace

extern "C" {

int wavemoth_shard_alm2map_legendre(wavemoth_plan plan, const double *alm, double *q_send, void *stream) {
  if (int rc = shard_check(plan, alm, q_send)) return rc;
  return finish(plan, run_legendre(plan, true, alm, nullptr, nullptr, q_origin(plan, q_send), (cudaStream_t)stream));
}

int wavemoth_shard_alm2map_rings(wavemoth_plan plan, const double *q_recv, double *q_ring, double *map,
                                 void *stream) {
  if (int rc = shard_check(plan, q_recv, q_ring)) return rc;
  if (!map) return set_error(WAVEMOTH_ERR_ARG, "NULL map");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nrl = plan->ring_bounds[plan->part + 1] - plan->ring_bounds[plan->part];
  int rc = cuda_check(wm::launch_shard_exchange(plan->d_shard_tab, nrl, plan->mmax + 1, plan->nvecs, q_recv, q_ring,
                                                1, st), "shard exchange");
  wm::RingParams r = ring_params(plan);
  r.q = ring_origin(plan, (const double *)q_ring);
  r.map = map;
  r.map_scale = 1.0;
  if (!rc) rc = cuda_check(wm::launch_ring_synthesis(r, st), "ring synthesis launch");
  plan->kernel_launches += 2;
  return finish(plan, rc);
}

int wavemoth_shard_map2alm_rings(wavemoth_plan plan, const double *map, double *q_ring, double *q_send,
                                 void *stream) {
  if (int rc = shard_check(plan, q_ring, q_send)) return rc;
  if (!map) return set_error(WAVEMOTH_ERR_ARG, "NULL map");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nrl = plan->ring_bounds[plan->part + 1] - plan->ring_bounds[plan->part];
  wm::RingParams r = ring_params(plan);
  r.map_in = map;
  r.q_out = ring_origin(plan, q_ring);
  int rc = cuda_check(wm::launch_ring_analysis(r, st), "ring analysis launch");
  if (!rc)
    rc = cuda_check(wm::launch_shard_exchange(plan->d_shard_tab, nrl, plan->mmax + 1, plan->nvecs, q_ring, q_send, 0,
                                              st), "shard exchange");
  plan->kernel_launches += 2;
  return finish(plan, rc);
}

int wavemoth_shard_map2alm_legendre(wavemoth_plan plan, const double *q_recv, double *alm, void *stream) {
  if (int rc = shard_check(plan, q_recv, alm)) return rc;
  return finish(plan, run_legendre(plan, false, nullptr, alm, q_origin(plan, q_recv), nullptr, (cudaStream_t)stream));
}

int wavemoth_legendre_alm2map_device(wavemoth_plan plan, const double *alm, double *q, void *stream) {
  if (int rc = whole_plan_check(plan, alm, q)) return rc;
  return finish(plan, run_legendre(plan, true, alm, nullptr, nullptr, q, (cudaStream_t)stream));
}

int wavemoth_legendre_map2alm_device(wavemoth_plan plan, const double *q, double *alm, void *stream) {
  if (int rc = whole_plan_check(plan, alm, q)) return rc;
  return finish(plan, run_legendre(plan, false, nullptr, alm, q, nullptr, (cudaStream_t)stream));
}

int wavemoth_plan_set_ring_weights(wavemoth_plan plan, const double *weights) {
  if (!plan) return set_error(WAVEMOTH_ERR_ARG, "NULL plan");
  if (plan->stream) cudaStreamSynchronize(plan->stream);
  if (!weights) {
    plan->d_ring_weights = nullptr;  // the buffer stays with the plan's arena
    return 0;
  }
  for (int r = 0; r < plan->ni; ++r)
    if (!(weights[r] > 0.0) || !std::isfinite(weights[r]))
      return set_error(WAVEMOTH_ERR_ARG, "ring weights must be positive and finite");
  static_assert(sizeof(double) == 8, "");
  if (!plan->d_ring_weights_buf)
    if (int rc = plan->arena.alloc(&plan->d_ring_weights_buf, (size_t)plan->ni, "ring weights")) return rc;
  if (int rc = cuda_check(cudaMemcpy(plan->d_ring_weights_buf, weights, (size_t)plan->ni * sizeof(double),
                                     cudaMemcpyHostToDevice), "ring weights upload"))
    return rc;
  plan->d_ring_weights = plan->d_ring_weights_buf;
  return 0;
}

int wavemoth_alm2map_backward_device(wavemoth_plan plan, const double *grad_map, double *grad_alm, void *stream) {
  if (int bad = whole_plan_check(plan, grad_map, grad_alm)) return bad;
  cudaStream_t st = (cudaStream_t)stream;
  const bool fused = weighs_alm(plan);
  int rc = run_map2alm(plan, grad_map, grad_alm, st, true, fused ? AlmOut::kBackward : AlmOut::kWrite);
  if (!rc && !fused) {
    rc = cuda_check(wm::launch_backward_weights(grad_alm, plan->lmax + 1, plan->nalm, plan->nvecs, st),
                    "backward weights");
    plan->kernel_launches++;
  }
  return finish(plan, rc);
}

int wavemoth_map2alm_iterative_device(wavemoth_plan plan, const double *map, double *alm, int niter,
                                      void *stream) {
  if (int bad = whole_plan_check(plan, map, alm)) return bad;
  if (niter < 0) return set_error(WAVEMOTH_ERR_ARG, "niter < 0");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nmap = plan->npix * plan->nmaps, nalm = plan->nalm * plan->nvecs;
  int rc = 0;
  const bool add = weighs_alm(plan);
  if (niter > 0 && !plan->d_iter_map) rc = plan->arena.alloc(&plan->d_iter_map, (size_t)nmap, "iteration map buffer");
  // (also when this call adds in place: a wait limit may change that later)
  if (niter > 0 && (plan->split || plan->nslow > 0) && !plan->d_iter_alm)
    rc = rc ? rc : plan->arena.alloc(&plan->d_iter_alm, (size_t)nalm, "iteration alm buffer");
  if (rc) return finish(plan, rc);
  rc = run_map2alm(plan, map, alm, st);
  for (int it = 0; it < niter && !rc; ++it) {
    // a += map2alm(f - alm2map(a))
    rc = run_alm2map(plan, alm, plan->d_iter_map, st, 1.0, map);
    if (!rc) rc = run_map2alm(plan, plan->d_iter_map, add ? alm : plan->d_iter_alm, st, false,
                              add ? AlmOut::kAdd : AlmOut::kWrite);
    if (rc || add) continue;
    rc = cuda_check(wm::launch_accumulate(plan->d_iter_alm, alm, nalm, st), "accumulate");
    plan->kernel_launches++;
  }
  return finish(plan, rc);
}

void wavemoth_perform_legendre_transforms(wavemoth_plan plan) {
  if (!plan) return;
  int rc = 0;
  if (plan->analysis) {
    rc = set_error(WAVEMOTH_ERR_ARG, "perform_legendre_transforms needs an alm2map plan");
  } else if (!plan->host_in) {
    rc = set_error(WAVEMOTH_ERR_ARG, "plan has no bound input buffer");
  } else if (plan->flags & WAVEMOTH_DEVICE_POINTERS) {
    rc = run_legendre(plan, true, plan->host_in, nullptr, nullptr, plan->d_q, plan->stream);
  } else {
    rc = cuda_check(cudaMemcpyAsync(plan->d_alm, plan->host_in,
                                    (size_t)plan->nalm * plan->nvecs * sizeof(double),
                                    cudaMemcpyHostToDevice, plan->stream),
                    "alm upload");
    rc = rc ? rc : run_legendre(plan, true, plan->d_alm, nullptr, nullptr, plan->d_q, plan->stream);
  }
  if (!rc) rc = cuda_check(cudaStreamSynchronize(plan->stream), "Legendre transforms");
  finish(plan, rc);
}

void wavemoth_perform_backward_ffts(wavemoth_plan plan) {
  if (!plan) return;
  int rc = 0;
  if (plan->analysis) {
    rc = set_error(WAVEMOTH_ERR_ARG, "perform_backward_ffts needs an alm2map plan");
  } else if (!plan->host_out) {
    rc = set_error(WAVEMOTH_ERR_ARG, "plan has no bound output buffer");
  } else {
    const bool devptr = (plan->flags & WAVEMOTH_DEVICE_POINTERS) != 0;
    wm::RingParams r = ring_params(plan);
    r.q = plan->d_q;
    r.map = devptr ? plan->host_out : plan->d_map;
    rc = cuda_check(wm::launch_ring_synthesis(r, plan->stream), "ring synthesis launch");
    plan->kernel_launches += r.ntasks > 0;
    if (!rc && !devptr)
      rc = cuda_check(cudaMemcpyAsync(plan->host_out, plan->d_map,
                                      (size_t)plan->npix * plan->nmaps * sizeof(double),
                                      cudaMemcpyDeviceToHost, plan->stream),
                      "map download");
    if (!rc) rc = cuda_check(cudaStreamSynchronize(plan->stream), "backward FFTs");
  }
  finish(plan, rc);
}

int wavemoth_plan_set_hemisphere_mode(wavemoth_plan plan, int one_side) {
  if (int rc = whole_plan_check(plan, plan, plan)) return rc;
  RingTable RT = ring_table(plan->nside, plan->nmaps, plan->mmax, one_side != 0);
  if (RT.max_cta_cplx > wm::kRingBufferCplx)
    return set_error(WAVEMOTH_ERR_ARG, "ring transforms longer than the CTA buffer");
  wm::DevRingTask *tasks = nullptr;
  if (int rc = upload(plan->arena, &tasks, RT.tasks, "ring work list")) return rc;
  if (plan->stream) cudaStreamSynchronize(plan->stream);
  plan->d_ring_tasks = tasks;
  plan->ring_ntasks = (int32_t)RT.tasks.size();
  plan->ring_smem = RT.smem;
  plan->ring_threads = RT.threads;
  plan->ring_short = RT.short_rings;
  return 0;
}

void wavemoth_disable_phase_shifting(wavemoth_plan plan) {
  if (plan) plan->phase_shifts = 0;
}

int wavemoth_get_work(wavemoth_plan plan, double *out) {
  if (int bad = whole_plan_check(plan, out, out)) return bad;
  const int64_t nrow = 2LL * (plan->mmax + 1) * plan->ni, nv = plan->nvecs;
  std::vector<double> dev((size_t)(nrow * nv));
  int rc = cuda_check(cudaMemcpyAsync(dev.data(), plan->d_q, dev.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                      plan->stream), "work download");
  if (!rc) rc = cuda_check(cudaStreamSynchronize(plan->stream), "work download");
  if (rc) return rc;
  // device rows are ring-major (wm::q_row); the reference's work_q is
  // (m, parity)-major: row (2m + parity) ni + ring
  for (int64_t r = 0; r < plan->ni; ++r)
    for (int m = 0; m <= plan->mmax; ++m)
      for (int odd = 0; odd < 2; ++odd)
        memcpy(out + ((2LL * m + odd) * plan->ni + r) * nv, dev.data() + wm::q_row(plan->mmax, m, odd, r) * nv,
               (size_t)nv * sizeof(double));
  return 0;
}

int wavemoth_plan_nmaps(wavemoth_plan plan) { return plan ? plan->nmaps : -1; }
int wavemoth_plan_nside(wavemoth_plan plan) { return plan ? plan->nside : -1; }
int wavemoth_plan_lmax(wavemoth_plan plan) { return plan ? plan->lmax : -1; }
int64_t wavemoth_plan_device_bytes(wavemoth_plan plan) { return plan ? plan->arena.base + plan->arena.bytes : -1; }
int64_t wavemoth_plan_program_bytes(wavemoth_plan plan) { return plan ? plan->img->program_bytes : -1; }
int64_t wavemoth_plan_image_bytes(wavemoth_plan plan) { return plan ? plan->img->arena.bytes : -1; }

void wavemoth_set_device_memory_cap(int64_t bytes) { g_device_cap = bytes; }

int wavemoth_plan_set_grid_cap(wavemoth_plan plan, int sms) {
  if (!plan || sms < 0) return set_error(WAVEMOTH_ERR_ARG, "wavemoth_plan_set_grid_cap: bad argument");
  plan->grid_cap = sms;
  return 0;
}

int wavemoth_plan_set_wait_limit(wavemoth_plan plan, int64_t polls) {
  if (!plan || polls < 0) return set_error(WAVEMOTH_ERR_ARG, "wavemoth_plan_set_wait_limit: bad argument");
  plan->wait_limit = polls;
  if (!plan->split || use_direct(plan) || plan->d_res_a) return 0;
  // a plan of few maps that is now to run the GEMMs.  Allocating and running on
  // the plan's own stream disturbs no capture, which the driver is told
  std::lock_guard<std::mutex> lock(g_image_mutex);
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  cudaThreadExchangeStreamCaptureMode(&mode);
  const int rc = provide_slices(plan);
  cudaThreadExchangeStreamCaptureMode(&mode);
  plan->arena.base = plan->img->arena.bytes;
  return rc;
}

int wavemoth_plan_route(wavemoth_plan plan) {
  if (!plan) return -1;
  return use_direct(plan) ? WAVEMOTH_ROUTE_FP64 : plan->d_res_a ? WAVEMOTH_ROUTE_GEMM : WAVEMOTH_ROUTE_GEMM_GENERATE;
}

int wavemoth_plan_timing(wavemoth_plan plan, int mode, double *out) {
  if (!plan) return set_error(WAVEMOTH_ERR_ARG, "NULL plan");
  if (mode == 0 || mode == 1) {
    if (plan->stream) cudaStreamSynchronize(plan->stream);
    for (auto &s : plan->spans) { cudaEventDestroy(s.a); cudaEventDestroy(s.b); }
    plan->spans.clear();
    plan->timing = (mode == 1);
    plan->kernel_launches = 0;
    return 0;
  }
  if (mode != 2 || !out) return set_error(WAVEMOTH_ERR_ARG, "invalid timing mode");
  for (int i = 0; i < 8; ++i) out[i] = 0.0;
  for (auto &s : plan->spans) {
    if (int rc = cuda_check(cudaEventSynchronize(s.b), "timing event")) return rc;
    float ms = 0.f;
    if (int rc = cuda_check(cudaEventElapsedTime(&ms, s.a, s.b), "timing event")) return rc;
    out[s.kind] += ms;
    out[4 + s.kind] += 1.0;
  }
  return 0;
}

int64_t wavemoth_plan_kernel_launches(wavemoth_plan plan) { return plan ? plan->kernel_launches : -1; }

int wavemoth_plan_work(wavemoth_plan plan, int nmaps, double *out) {
  if (!plan || !out || nmaps <= 0) return set_error(WAVEMOTH_ERR_ARG, "invalid arguments");
  const auto &G = plan->img->prog;
  const double nvecs = 2.0 * nmaps;
  // Legendre: multiply-adds of the interpolation and residual products, plus
  // 5 flops per recurrence element (shared by all vectors)
  out[0] = 2.0 * nvecs * (double)(G.interp_elems + G.rec_elems + G.dense_elems) + 5.0 * (double)G.rec_elems;
  // compressed-matrix bytes one direction streams: interpolants (one copy),
  // dense residual values, x2/P0/P1 per recurrence column, coefficients
  out[1] = 8.0 * (double)(G.interp_elems + G.dense_elems + 3 * G.rec_columns + G.aux_values);
  // vector traffic of one Legendre launch: alm in (or out) and q out (or in)
  const double nalm = (double)plan->nalm, nq = 2.0 * (plan->mmax + 1) * plan->ni;
  out[2] = 8.0 * nvecs * (nalm + nq);
  // ring kernels: q in (or out) and the maps out (or in)
  out[3] = 8.0 * (nvecs * nq + (double)plan->npix * nmaps);
  out[4] = (double)G.interp_elems;
  out[5] = (double)G.rec_elems;
  out[6] = (double)G.dense_elems;
  out[7] = (double)plan->grid;
  out[8] = out[9] = out[10] = out[11] = 0.0;
  if (use_direct(plan)) return 0;
  // split path: 64-row (or 64-column) K chunks of 128-row M tiles; per K
  // step of 32, nine MMAs with N summing to 1664 (six slices, i + j <= 6)
  double ea = 0.0, eb = 0.0, la = 0.0, lb = 0.0;
  for (const auto &T : G.stiles_a) ea += (double)(G.sgroups[T.group].nrchunks - T.kc0);
  for (const auto &T : G.stiles_b) eb += (double)T.nk;
  for (const auto &T : G.stiles_la) la += (double)G.sroots[T.unit].nsc;
  for (const auto &T : G.stiles_lm) lb += (double)G.sroots[T.unit].nzc;
  const double chunk = (double)wm::kSplitM * wm::kSplitK;
  const double passes = (double)((2 * nmaps + wm::kSplitN - 1) / wm::kSplitN);
  const double ops_per_elem = 2.0 * 1664.0;  // per element of an A chunk (M x K), all slice windows
  out[8] = ea * chunk;
  out[9] = eb * chunk;
  out[10] = (ea + la) * chunk * ops_per_elem * passes;
  out[11] = (eb + lb) * chunk * ops_per_elem * passes;
  return 0;
}

int wavemoth_check_resourcefile(char *filename, int Nside, int lmax, int64_t *out_stats) {
  if (!filename) return set_error(WAVEMOTH_ERR_ARG, "NULL file name");
  std::vector<char> file;
  std::string err;
  if (!read_file(filename, file, err)) return set_error(WAVEMOTH_ERR_RESOURCE, err);
  wm::HostProgram P;
  if (!wm::compile_resource(file.data(), file.size(), Nside, lmax, lmax, P, err))
    return set_error(WAVEMOTH_ERR_RESOURCE, std::string(filename) + ": " + err);
  if (!wm::build_fast_path(P, false, err))
    return set_error(WAVEMOTH_ERR_RESOURCE, std::string(filename) + ": " + err);
  if (out_stats) {
    out_stats[0] = (int64_t)P.mats.size();
    out_stats[1] = (int64_t)P.dblocks.size();
    out_stats[2] = (int64_t)P.strips.size();
    out_stats[3] = (int64_t)P.levels.size();
    out_stats[4] = (int64_t)P.pairs.size();
    out_stats[5] = (int64_t)P.f64.size() * 8;
    out_stats[6] = (int64_t)P.i32.size() * 4;
    out_stats[7] = P.max_rows;
  }
  return 0;
}

wavemoth_grid_info *wavemoth_create_healpix_grid_info(int Nside) {
  if (Nside <= 0 || Nside > (1 << 13)) {
    set_error(WAVEMOTH_ERR_ARG, "invalid Nside");
    return nullptr;
  }
  const int nrings = 4 * Nside - 1;
  char *buf = (char *)malloc(sizeof(wavemoth_grid_info) + sizeof(double) * nrings +
                             sizeof(bfm_index_t) * (nrings + 1));
  if (!buf) return nullptr;
  auto *g = (wavemoth_grid_info *)buf;
  g->phi0s = (double *)(buf + sizeof(wavemoth_grid_info));
  g->ring_offsets = (bfm_index_t *)(g->phi0s + nrings);
  g->has_equator = 1;
  g->nrings = nrings;
  g->mid_ring = 2 * Nside - 1;
  int npr = 0, ipix = 0;
  const double pi = 3.14159265358979323846;
  for (int r = 0; r < nrings; ++r) {
    if (r <= Nside - 1) {
      npr += 4;
      g->phi0s[r] = pi / (4.0 * (r + 1));
    } else if (r > 3 * Nside - 1) {
      npr -= 4;
      g->phi0s[r] = pi / (4.0 * (nrings - r));
    } else {
      g->phi0s[r] = (pi / (4.0 * Nside)) * (r % 2);
    }
    g->ring_offsets[r] = ipix;
    ipix += npr;
  }
  g->ring_offsets[nrings] = ipix;
  g->npix = ipix;
  return g;
}

void wavemoth_free_grid_info(wavemoth_grid_info *info) { free(info); }

}  // extern "C"
