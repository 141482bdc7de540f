// Harness kernels on the device: the analytic right-hand side (FishFry.hpp:14-45)
// with an optional seeded sum of Fourier modes, and the error sums against the
// analytic solution (FishFry.hpp:47-101) with a deterministic reduction in
// place of the reference's shared and global FP64 atomics.

#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "ff_status.hpp"

namespace ff {

constexpr int kMaxModes = 64;
constexpr int kSumBlocks = 1184;   // 8 blocks per SM on 148 SMs; fixed, so sums are reproducible
constexpr int kSumThreads = 256;

struct FieldArgs {
  int ni, nj, nk;
  double xlo, ylo, zlo, dx, dy, dz;
  int nmodes;
  int finite;   // every amplitude is
  ff_mode modes[kMaxModes];
};

// Weight of a mode in f or in phi; the zero mode counts as absent.
__device__ __forceinline__ int mode_k2(const ff_mode &m) { return m.kx * m.kx + m.ky * m.ky + m.kz * m.kz; }
__device__ __forceinline__ double mode_weight(const ff_mode &m, bool solution) {
  return solution ? -m.a / (double)mode_k2(m) : m.a;
}

// phi factors and their second derivatives along one axis, FishFry.hpp:22-41
// and :71-86: (factor, second derivative) at one coordinate.
__device__ __forceinline__ double2 factor_x(double x) {
  const double cx = cos(x), sx = sin(x), ex = exp(sx);
  return make_double2(cx * ex, -ex * sx * cx * (sx + 3.0));
}
__device__ __forceinline__ double2 factor_y(double y) {
  const double cy = cos(y), sy = sin(y), ey = exp(cy);
  return make_double2(sy * ey, sy * ey * (sy * sy - 3.0 * cy - 1.0));
}
__device__ __forceinline__ double2 factor_z(double z) {
  const double cz = cos(z), sz = sin(z), ez = exp(cz);
  return make_double2(cz * ez, ez * (3.0 * sz * sz - cz * cz * cz - 1.0));
}

// Both field kernels walk tiles of kTileLines (i, j) lines by at most kTileK
// points along z.  f and phi are sums of products of one-axis factors, and a
// mode's cosine is cos(A + B) = cos A cos B - sin A sin B with A = kx x + ky y
// + theta of the line and B = kz z of the point, so a tile evaluates sines,
// cosines and exponentials once per line and once per k, in shared memory,
// and a point costs its products and two multiply-adds per mode, not nine FP64
// transcendentals (and one more per mode).  Tables and FP64 arithmetic bound the
// kernels, not HBM: 256^3 FP64 without modes k_init takes 27 us for 21 us of
// writes, k_diff 35 us with phi and 33 without reading it.  f and both norms (three
// calls) point by point 1.67-1.97 ms, so 0.145 ms, of which about 0.06 ms is launch
// and wait latency.  Grids whose tiles would be mostly empty go point by point
// (by_points).
//
// A block keeps its z chunk (blockIdx.x % columns) and walks the line tiles, so
// the z tables are formed once per block (once per chunk on lines of more than
// kSumBlocks chunks).  Thread (w, lane) holds lines
// 8w .. 8w+7 of the tile at k = lane and lane + 32: its 16 points share 8 line
// and 2 z table entries per mode, in registers.
constexpr int kTileLines = 64;
constexpr int kTileK = 64;
constexpr int kTileWarpLines = kTileLines / (kSumThreads / 32);

struct FieldTiles {
  long tiles;     // line tiles
  int chunks;     // z chunks of kc points
  int kc;
  int columns;    // blocks side by side along the chunks (at most kSumBlocks)
  int walkers;    // blocks per column, sharing its line tiles
};

// Values of the tile's 16 points of this thread: f (solution = false) or phi,
// summed as the point-by-point formulas are (FishFry.hpp:44, :87).
template <bool MODES>
__device__ __forceinline__ void tile_values(const FieldArgs &a, const double2 *sm, int warp, int lane, bool solution,
                                            double v[kTileWarpLines][2]) {
  const double2 *zf = sm, *lx = sm + kTileK, *ly = lx + kTileLines;
  const double2 *zm = ly + kTileLines, *lm = zm + a.nmodes * kTileK;
  const double2 z[2] = {zf[lane], zf[lane + 32]};
#pragma unroll
  for (int l = 0; l < kTileWarpLines; l++) {
    const double2 x = lx[warp * kTileWarpLines + l], y = ly[warp * kTileWarpLines + l];
#pragma unroll
    for (int q = 0; q < 2; q++)
      v[l][q] = solution ? x.x * y.x * z[q].x : x.x * y.x * z[q].y + x.x * y.y * z[q].x + x.y * y.x * z[q].x;
  }
  if constexpr (!MODES) return;
  double s[kTileWarpLines][2] = {};
  for (int m = 0; m < a.nmodes; m++) {
    const double2 b0 = zm[m * kTileK + lane], b1 = zm[m * kTileK + lane + 32];
#pragma unroll
    for (int l = 0; l < kTileWarpLines; l++) {
      const double2 w = lm[m * kTileLines + warp * kTileWarpLines + l];   // weight times (cos A, sin A)
      s[l][0] = fma(w.x, b0.x, s[l][0]);
      s[l][1] = fma(w.x, b1.x, s[l][1]);
      s[l][0] = fma(-w.y, b0.y, s[l][0]);
      s[l][1] = fma(-w.y, b1.y, s[l][1]);
    }
  }
#pragma unroll
  for (int l = 0; l < kTileWarpLines; l++) {
    v[l][0] += s[l][0];
    v[l][1] += s[l][1];
  }
}

// z tables of a chunk (once per block) and line tables of a line tile.
// Entries past the chunk or the grid repeat its last point; they are not used.
__device__ __forceinline__ void z_tables(const FieldArgs &a, double2 *sm, int k0, int kc) {
  double2 *zf = sm, *zm = sm + kTileK + 2 * kTileLines;
  for (int q = threadIdx.x; q < kTileK * (1 + a.nmodes); q += kSumThreads) {
    const int k = k0 + min(q % kTileK, kc - 1);
    const double z = a.zlo + k * a.dz;
    if (q < kTileK) {
      zf[q] = factor_z(z);
    } else {
      const int m = q / kTileK - 1;
      double2 b;
      sincos((double)a.modes[m].kz * z, &b.y, &b.x);
      zm[q - kTileK] = b;
    }
  }
}
__device__ __forceinline__ void line_tables(const FieldArgs &a, double2 *sm, long line0, long nlines, bool solution) {
  double2 *lx = sm + kTileK, *ly = lx + kTileLines, *lm = ly + kTileLines + a.nmodes * kTileK;
  for (int q = threadIdx.x; q < kTileLines * (2 + a.nmodes); q += kSumThreads) {
    const long line = min(line0 + q % kTileLines, nlines - 1);
    const int i = (int)(line / a.nj);
    const int j = (int)(line - (long)i * a.nj);
    const double x = a.xlo + i * a.dx, y = a.ylo + j * a.dy;
    if (q < kTileLines) {
      lx[q] = factor_x(x);
    } else if (q < 2 * kTileLines) {
      ly[q - kTileLines] = factor_y(y);
    } else {
      // weight a (f) or -a / |k|^2 (phi) times the line's cosine and sine
      const ff_mode &md = a.modes[q / kTileLines - 2];
      double2 v = make_double2(0.0, 0.0);
      if (mode_k2(md) != 0) {
        const double w = mode_weight(md, solution);
        sincos((double)md.kx * x + (double)md.ky * y + md.theta, &v.y, &v.x);
        v = make_double2(w * v.x, w * v.y);
      }
      lm[q - 2 * kTileLines] = v;
    }
  }
}

template <typename T, bool MODES>
__global__ void __launch_bounds__(kSumThreads, MODES ? 2 : 4) k_init(const FieldArgs a, const FieldTiles t, T *__restrict__ f) {
  extern __shared__ double2 smf[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const long nlines = (long)a.ni * a.nj;
  for (int chunk = blockIdx.x % t.columns; chunk < t.chunks; chunk += t.columns) {
    const int k0 = chunk * t.kc, kc = min(t.kc, a.nk - k0);
    __syncthreads();
    z_tables(a, smf, k0, kc);
    for (long tile = blockIdx.x / t.columns; tile < t.tiles; tile += t.walkers) {
      const long line0 = tile * kTileLines;
      __syncthreads();
      line_tables(a, smf, line0, nlines, false);
      __syncthreads();
      double v[kTileWarpLines][2];
      tile_values<MODES>(a, smf, warp, lane, false, v);
#pragma unroll
      for (int l = 0; l < kTileWarpLines; l++) {
        const long line = line0 + warp * kTileWarpLines + l;
        if (line >= nlines) break;
        T *row = f + line * a.nk + k0;
        if (lane < kc) row[lane] = (T)v[l][0];
        if (lane + 32 < kc) row[lane + 32] = (T)v[l][1];
      }
    }
  }
}

// f (solution = false) or phi at point q by the formulas as they stand.
__device__ __forceinline__ double point_value(const FieldArgs &a, long q, bool solution) {
  const long line = q / a.nk;
  const int k = (int)(q - line * a.nk);
  const int i = (int)(line / a.nj);
  const int j = (int)(line - (long)i * a.nj);
  const double x = a.xlo + i * a.dx, y = a.ylo + j * a.dy, z = a.zlo + k * a.dz;
  const double2 px = factor_x(x), py = factor_y(y), pz = factor_z(z);
  double v = solution ? px.x * py.x * pz.x   // FishFry.hpp:87, :44
                      : px.x * py.x * pz.y + px.x * py.y * pz.x + px.y * py.x * pz.x;
  if (a.nmodes == 0) return v;
  double s = 0.0;
  for (int m = 0; m < a.nmodes; m++) {
    const ff_mode &md = a.modes[m];
    if (mode_k2(md) == 0) continue;
    s += mode_weight(md, solution) * cos((double)md.kx * x + (double)md.ky * y + (double)md.kz * z + md.theta);
  }
  return v + s;
}

// Point by point, in place of the tiles' kernels (by_points).
template <typename T> __global__ void __launch_bounds__(kSumThreads) k_init_points(const FieldArgs a, T *__restrict__ f) {
  const long N = (long)a.ni * a.nj * a.nk;
  for (long q = blockIdx.x * (long)kSumThreads + threadIdx.x; q < N; q += (long)gridDim.x * kSumThreads)
    f[q] = (T)point_value(a, q, false);
}

// One point's difference (FishFry.hpp:89) into a thread's {sum|d|, sum d^2,
// max|d|}.  NaN propagates through the max, as the reference's integer atomicMax
// on the bit pattern does.
struct DiffSums {
  double t1 = 0, t2 = 0, tm = 0;
  __device__ __forceinline__ void add(double exact, double phi) {
    const double d = fabs(exact - phi);
    t1 += d;
    t2 += d * d;
    tm = (d > tm || d != d) ? d : tm;
  }
};

// The block's sums in a fixed tree, into out[0..2].
__device__ __forceinline__ void block_sums(const DiffSums &t, double *out) {
  __shared__ double s1[kSumThreads], s2[kSumThreads], sm[kSumThreads];
  s1[threadIdx.x] = t.t1;
  s2[threadIdx.x] = t.t2;
  sm[threadIdx.x] = t.tm;
  __syncthreads();
  for (int w = kSumThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      s1[threadIdx.x] += s1[threadIdx.x + w];
      s2[threadIdx.x] += s2[threadIdx.x + w];
      const double o = sm[threadIdx.x + w];
      if (o > sm[threadIdx.x] || o != o) sm[threadIdx.x] = o;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = s1[0];
    out[1] = s2[0];
    out[2] = sm[0];
  }
}

template <typename T>
__global__ void __launch_bounds__(kSumThreads) k_diff_points(const FieldArgs a, const T *__restrict__ phi,
                                                             double *__restrict__ partial) {
  const long N = (long)a.ni * a.nj * a.nk;
  DiffSums t;
  for (long q = blockIdx.x * (long)kSumThreads + threadIdx.x; q < N; q += (long)gridDim.x * kSumThreads)
    t.add(point_value(a, q, true), phi ? (double)phi[q] : 0.0);
  block_sums(t, partial + 3 * blockIdx.x);
}

// Stage 1 of the error sums: per-block {sum|d|, sum d^2, max|d|} over the
// block's tiles, each thread's points in a fixed order, reduced in a fixed
// tree; the grid is a function of the dimensions alone, so the sums are
// reproducible.
template <typename T, bool MODES>
__global__ void __launch_bounds__(kSumThreads, MODES ? 2 : 3) k_diff(const FieldArgs a, const FieldTiles t, const T *__restrict__ phi,
                                                      double *__restrict__ partial) {
  extern __shared__ double2 smf[];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const long nlines = (long)a.ni * a.nj;
  DiffSums sums;
  for (int chunk = blockIdx.x % t.columns; chunk < t.chunks; chunk += t.columns) {
    const int k0 = chunk * t.kc, kc = min(t.kc, a.nk - k0);
    __syncthreads();
    z_tables(a, smf, k0, kc);
    for (long tile = blockIdx.x / t.columns; tile < t.tiles; tile += t.walkers) {
      const long line0 = tile * kTileLines;
      // the tile's phi first: its loads are in flight while the tables are formed
      T p[kTileWarpLines][2];
#pragma unroll
      for (int l = 0; l < kTileWarpLines; l++) {
        const long line = line0 + warp * kTileWarpLines + l;
        const T *row = phi + line * a.nk + k0;
        p[l][0] = phi && line < nlines && lane < kc ? row[lane] : (T)0;
        p[l][1] = phi && line < nlines && lane + 32 < kc ? row[lane + 32] : (T)0;
      }
      __syncthreads();
      line_tables(a, smf, line0, nlines, true);
      __syncthreads();
      double v[kTileWarpLines][2];
      tile_values<MODES>(a, smf, warp, lane, true, v);
#pragma unroll
      for (int l = 0; l < kTileWarpLines; l++) {
        const long line = line0 + warp * kTileWarpLines + l;
#pragma unroll
        for (int q = 0; q < 2; q++) {
          if (line < nlines && lane + 32 * q < kc) sums.add(v[l][q], (double)p[l][q]);
        }
      }
    }
  }
  block_sums(sums, partial + 3 * blockIdx.x);
}

// Stage 2: one block folds the per-block partials in a fixed order.
__global__ void __launch_bounds__(kSumThreads) k_diff_final(const double *__restrict__ partial, int nb,
                                                            double *__restrict__ out) {
  DiffSums t;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    t.t1 += partial[3 * b];
    t.t2 += partial[3 * b + 1];
    const double o = partial[3 * b + 2];
    t.tm = (o > t.tm || o != o) ? o : t.tm;
  }
  block_sums(t, out);
}

static int field_args(const int n[3], const double xlo[3], const double dx[3], int nmodes, const ff_mode *modes,
                      FieldArgs &a) {
  if (!n || !xlo || !dx) return set_error(FF_ERR_INVALID, "null argument");
  for (int d = 0; d < 3; d++)
    if (n[d] < 1) return set_error(FF_ERR_INVALID, "n[%d] = %d < 1", d, n[d]);
  if (nmodes < 0 || nmodes > kMaxModes || (nmodes > 0 && !modes))
    return set_error(FF_ERR_INVALID, "nmodes = %d outside [0, %d]", nmodes, kMaxModes);
  std::memset(&a, 0, sizeof(a));
  a.ni = n[0];
  a.nj = n[1];
  a.nk = n[2];
  a.xlo = xlo[0];
  a.ylo = xlo[1];
  a.zlo = xlo[2];
  a.dx = dx[0];
  a.dy = dx[1];
  a.dz = dx[2];
  a.nmodes = nmodes;
  a.finite = 1;
  for (int m = 0; m < nmodes; m++) {
    a.modes[m] = modes[m];
    if (!std::isfinite(modes[m].a)) a.finite = 0;
  }
  return FF_OK;
}

// Launch shape: z chunks of equal length up to kTileK, and as many blocks per
// chunk as keep the grid within kSumBlocks (8 blocks per SM; one block per SM
// fits when 64 modes fill its tables).
static FieldTiles tile_shape(const FieldArgs &a) {
  FieldTiles t;
  const long nlines = (long)a.ni * a.nj;
  t.chunks = (a.nk + kTileK - 1) / kTileK;
  t.kc = (a.nk + t.chunks - 1) / t.chunks;
  t.chunks = (a.nk + t.kc - 1) / t.kc;
  t.columns = t.chunks < kSumBlocks ? t.chunks : kSumBlocks;
  t.tiles = (nlines + kTileLines - 1) / kTileLines;
  const int per_column = kSumBlocks / t.columns;
  t.walkers = per_column < t.tiles ? per_column : (int)t.tiles;
  return t;
}

// Whether a kernel goes point by point: for amplitudes that are not finite (a
// weight times cos A cos B - sin A sin B would be inf - inf), and where tiles hold so
// few points that their tables cost more than the points' own factors and
// cosines.  Points of a tile below which that is so, with 64 lines and a few points
// along z (12 million points FP64, tiles / points): the right-hand side without
// modes 3 points 235 / 223 us, 4 178 / 223; 16 modes 5 points 796 / 725, 6 667 / 725;
// 64 modes 7 points 2339 / 2214, 8 2054 / 2213; the sums without modes 4 points
// 284 / 252, 5 235 / 252, with 64 modes 6 3462 / 3152, 7 2983 / 3153.  A few long
// lines, whose chunks form the z tables anew, need a quarter more points: 64 modes 9
// lines 2293 / 2213, 10 2067 / 2213.  One line or one point along z takes up to nine
// times as long in tiles.
static bool by_points(const FieldArgs &a, const FieldTiles &t, bool sums) {
  const long nlines = (long)a.ni * a.nj;
  const long points = nlines < kTileLines ? t.kc * nlines * 4 / 5 : t.kc * kTileLines;
  const long least = a.nmodes == 0 ? (sums ? 260 : 200) : sums ? 340 + a.nmodes : 330 + a.nmodes * 14 / 5;
  return !a.finite || points < least;
}
// Their grid: up to `most` blocks.
static unsigned point_blocks(const FieldArgs &a, int most) {
  const long want = ((long)a.ni * a.nj * a.nk + kSumThreads - 1) / kSumThreads;
  return (unsigned)(want < most ? want : most);
}

static size_t tile_smem(const FieldArgs &a) {
  return sizeof(double2) * ((size_t)(1 + a.nmodes) * kTileK + (size_t)(2 + a.nmodes) * kTileLines);
}

// Lets fn use the tables of kMaxModes modes.
template <typename F> static int allow_tables(F fn, size_t smem) {
  if (smem > 48 * 1024 - 3 * kSumThreads * sizeof(double))
    FF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(double2) * ((1 + kMaxModes) * kTileK + (2 + kMaxModes) * kTileLines))));
  return FF_OK;
}

// Per-block partial sums of |exact phi - phi| into partial[3 * blocks].
static int launch_diff(const FieldArgs &a, int precision, const void *phi, double *partial, cudaStream_t st,
                       int *blocks) {
  const FieldTiles t = tile_shape(a);
  const size_t smem = tile_smem(a);
  const bool points = by_points(a, t, true);
  *blocks = points ? (int)point_blocks(a, kSumBlocks) : t.columns * t.walkers;
  auto launch = [&](auto fn, auto *p) -> int {
    const int rc = allow_tables(fn, smem);
    if (rc == FF_OK) fn<<<*blocks, kSumThreads, smem, st>>>(a, t, p, partial);
    return rc;
  };
  auto run = [&](auto *p) -> int {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(p)>>;
    if (!points) return a.nmodes > 0 ? launch(k_diff<T, true>, p) : launch(k_diff<T, false>, p);
    k_diff_points<T><<<*blocks, kSumThreads, 0, st>>>(a, p, partial);
    return FF_OK;
  };
  const int rc = precision == FF_FP64 ? run(static_cast<const double *>(phi)) : run(static_cast<const float *>(phi));
  if (rc != FF_OK) return rc;
  FF_CUDA(cudaGetLastError());
  return FF_OK;
}

// Scratch of ff_error_sums: the partial triples and the final triple of one
// call.  kSumSlots of them per GPU are part of the module; a call claims one for
// its duration (it waits for its stream before it returns, so the slot is idle
// again) and only allocates when all are in use by other threads.  An allocation
// per call cost more than the kernel: freed memory goes back to the system at the
// wait, and the next call maps it again (0.4 ms of a 0.8 ms call at 256^3).
constexpr int kSumSlots = 16;
constexpr int kSumSlotDoubles = 3 * kSumBlocks + 3;
static __device__ __align__(256) double g_sum_slots[kSumSlots][kSumSlotDoubles];

class SumScratch {
 public:
  explicit SumScratch(cudaStream_t st) : st_(st) {}
  ~SumScratch() {
    if (own_) cudaFreeAsync(p_, st_);
    if (slot_ >= 0) busy(dev_).fetch_and(~(1u << slot_));
  }
  SumScratch(const SumScratch &) = delete;
  SumScratch &operator=(const SumScratch &) = delete;
  int take(double **out) {
    FF_CUDA(cudaGetDevice(&dev_));
    if (dev_ >= 0 && dev_ < kDevices) {
      for (int q = 0; q < kSumSlots && slot_ < 0; q++)
        if (!(busy(dev_).fetch_or(1u << q) & (1u << q))) slot_ = q;
    }
    if (slot_ >= 0) {
      void *base = nullptr;
      FF_CUDA(cudaGetSymbolAddress(&base, g_sum_slots));
      *out = static_cast<double *>(base) + (size_t)slot_ * kSumSlotDoubles;
      return FF_OK;
    }
    FF_CUDA(cudaMallocAsync(reinterpret_cast<void **>(&p_), kSumSlotDoubles * sizeof(double), st_));
    own_ = true;
    *out = p_;
    return FF_OK;
  }

 private:
  static constexpr int kDevices = 64;
  static std::atomic<unsigned> &busy(int dev) {
    static std::atomic<unsigned> mask[kDevices] = {};
    return mask[dev];
  }
  cudaStream_t st_;
  int dev_ = -1, slot_ = -1;
  bool own_ = false;
  double *p_ = nullptr;
};

// ---------------------------------------------------------------------------
// Error sums without any device allocation.
//
// Some callers cannot allocate device memory at the point where they want the
// error norms: a host application whose own pool allocator has already
// reserved the device memory, a time-critical loop where cudaMalloc's implicit
// device synchronisation is not acceptable, or plug-in code that may not call
// the CUDA allocator at all.  For them the partial sums live in a fixed
// file-scope device array of their own instead of the slots or a per-call buffer:
// every GPU that loads this library holds it (28 KB) until the process exits.
//
// The kernels and the summation order are those of ff_error_sums.  kNoAllocMaxPoints
// = 2^30 points (1024^3) is the entry point's stated limit; the partials of
// kSumBlocks blocks would serve any grid.
constexpr long kNoAllocMaxPoints = 1L << 30;
static __device__ __align__(256) double g_noalloc_partials[kSumSlotDoubles];

// Device address of g_noalloc_partials on the current device.  The name is a
// host-side stand-in, not a device address, so it is looked up once per
// device (with that device current) and remembered.  A cudaDeviceReset in the
// process makes the remembered address stale (the module is reloaded, perhaps
// elsewhere): the entry point is not for use after a reset.
static int noalloc_partials(double **out) {
  static std::mutex mu;
  static void *addr[256] = {};
  int dev = 0;
  FF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) return set_error(FF_ERR_INVALID, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_partials);
    if (e != cudaSuccess)
      return set_error(FF_ERR_CUDA, "cudaGetSymbolAddress of the static partial-sum array failed: %s",
                       cudaGetErrorString(e));
    addr[dev] = p;
  }
  *out = static_cast<double *>(addr[dev]);
  return FF_OK;
}

}  // namespace ff

using namespace ff;

extern "C" {

int ff_init_field(const int n[3], const double xlo[3], const double dx[3], int nmodes, const ff_mode *modes,
                  int precision, void *f, void *stream) {
  FieldArgs a;
  int rc = field_args(n, xlo, dx, nmodes, modes, a);
  if (rc != FF_OK) return rc;
  if (!f) return set_error(FF_ERR_INVALID, "ff_init_field: null field");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision != FF_FP64 && precision != FF_FP32)
    return set_error(FF_ERR_INVALID, "ff_init_field: bad precision %d", precision);
  const FieldTiles t = tile_shape(a);
  const size_t smem = tile_smem(a);
  auto launch = [&](auto fn, auto *p) -> int {
    const int rc = allow_tables(fn, smem);
    if (rc == FF_OK) fn<<<t.columns * t.walkers, kSumThreads, smem, st>>>(a, t, p);
    return rc;
  };
  auto run = [&](auto *p) -> int {
    using T = std::remove_pointer_t<decltype(p)>;
    if (!by_points(a, t, false)) return a.nmodes > 0 ? launch(k_init<T, true>, p) : launch(k_init<T, false>, p);
    k_init_points<T><<<point_blocks(a, 8 * kSumBlocks), kSumThreads, 0, st>>>(a, p);
    return FF_OK;
  };
  rc = precision == FF_FP64 ? run(static_cast<double *>(f)) : run(static_cast<float *>(f));
  if (rc != FF_OK) return rc;
  FF_CUDA(cudaGetLastError());
  return FF_OK;
}

int ff_error_sums(const int n[3], const double xlo[3], const double dx[3], int nmodes, const ff_mode *modes,
                  int precision, const void *phi, double sums[3], void *stream) {
  FieldArgs a;
  int rc = field_args(n, xlo, dx, nmodes, modes, a);
  if (rc != FF_OK) return rc;
  if (!sums) return set_error(FF_ERR_INVALID, "ff_error_sums: null sums");
  if (precision != FF_FP64 && precision != FF_FP32)
    return set_error(FF_ERR_INVALID, "ff_error_sums: bad precision %d", precision);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  SumScratch held(st);
  double *scratch = nullptr;
  rc = held.take(&scratch);
  if (rc != FF_OK) return rc;
  int blocks = 0;
  rc = launch_diff(a, precision, phi, scratch, st, &blocks);
  if (rc != FF_OK) return rc;
  k_diff_final<<<1, kSumThreads, 0, st>>>(scratch, blocks, scratch + 3 * kSumBlocks);
  cudaError_t e = cudaGetLastError();
  double host[3] = {0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, scratch + 3 * kSumBlocks, sizeof(host), cudaMemcpyDeviceToHost, st);
  // the scratch is given back (and host read) only when the stream is done with it
  const cudaError_t es = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess)
    return set_error(FF_ERR_CUDA, "ff_error_sums: %s (%s)", cudaGetErrorName(e), cudaGetErrorString(e));
  sums[0] = host[0];
  sums[1] = host[1];
  sums[2] = host[2];
  return FF_OK;
}

int ff_error_sums_noalloc(const int n[3], const double xlo[3], const double dx[3], int nmodes,
                          const ff_mode *modes, int precision, const void *phi, double sums[3], void *stream) {
  FieldArgs a;
  int rc = field_args(n, xlo, dx, nmodes, modes, a);
  if (rc != FF_OK) return rc;
  if (!sums) return set_error(FF_ERR_INVALID, "ff_error_sums_noalloc: null sums");
  if (precision != FF_FP64 && precision != FF_FP32)
    return set_error(FF_ERR_INVALID, "ff_error_sums_noalloc: bad precision %d", precision);
  const long N = (long)n[0] * n[1] * n[2];
  if (N > kNoAllocMaxPoints)
    return set_error(FF_ERR_UNSUPPORTED,
                     "ff_error_sums_noalloc: %ld points are above this entry point's limit of %ld points", N,
                     kNoAllocMaxPoints);
  double *partial = nullptr;
  rc = noalloc_partials(&partial);
  if (rc != FF_OK) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // every slot read below is written by this call first: nothing to clear
  int blocks = 0;
  rc = launch_diff(a, precision, phi, partial, st, &blocks);
  if (rc != FF_OK) return rc;
  double *total = partial + 3 * kSumBlocks;
  k_diff_final<<<1, kSumThreads, 0, st>>>(partial, blocks, total);
  cudaError_t e = cudaGetLastError();
  double host[3] = {0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(host, total, sizeof(host), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess)
    return set_error(FF_ERR_CUDA, "ff_error_sums_noalloc: %s (%s)", cudaGetErrorName(e), cudaGetErrorString(e));
  sums[0] = host[0];
  sums[1] = host[1];
  sums[2] = host[2];
  return FF_OK;
}

// SplitMix64 (Steele, Lea and Flood, OOPSLA 2014) as a counter stream, and
// Box-Muller for the normal amplitudes.
int ff_modes_generate(uint64_t seed, int count, int kmax, const int kaxis[3], double sigma, ff_mode *out) {
  if (count < 0 || (count > 0 && !out) || !kaxis) return set_error(FF_ERR_INVALID, "ff_modes_generate: bad argument");
  uint64_t s = seed;
  auto next = [&]() {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  auto uniform = [&]() { return (double)(next() >> 11) * 0x1.0p-53; };
  const long kmax2 = (long)kmax * kmax;
  const bool possible = kmax > 0 && (kaxis[0] > 0 || kaxis[1] > 0 || kaxis[2] > 0);
  for (int m = 0; m < count; m++) {
    ff_mode md{0, 0, 0, 0.0, 0.0};
    if (possible) {
      for (;;) {
        const int kx = (int)(next() % (uint64_t)(2 * kaxis[0] + 1)) - kaxis[0];
        const int ky = (int)(next() % (uint64_t)(2 * kaxis[1] + 1)) - kaxis[1];
        const int kz = (int)(next() % (uint64_t)(2 * kaxis[2] + 1)) - kaxis[2];
        const long k2 = (long)kx * kx + (long)ky * ky + (long)kz * kz;
        if (k2 == 0 || k2 > kmax2) continue;
        md.kx = kx;
        md.ky = ky;
        md.kz = kz;
        break;
      }
      const double u1 = 1.0 - uniform();
      const double u2 = uniform();
      md.a = sigma * std::sqrt(-2.0 * std::log(u1)) * std::cos(2.0 * M_PI * u2);
      md.theta = 2.0 * M_PI * uniform();
    }
    out[m] = md;
  }
  return FF_OK;
}

}  // extern "C"
