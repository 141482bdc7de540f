// Device code of the batch passes: grid descriptors, the column tiles of the
// strided passes, the per-pass kernel and its launch helpers.
// Included by ff_batch_f64.cu and ff_batch_f32.cu, one precision each.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstring>

#include "ff_batch.hpp"
#include "ff_gen_lines.cuh"
#include "ff_status.hpp"
#include "ff_tiles.cuh"

namespace ff {

// Device descriptor of one grid: its pass arguments and buffers, and per pass the
// tile shape and, for runtime plans, the stages as the tiles walk them.  The head
// and the pass's part are copied into shared memory for each tile.
struct alignas(16) KindDesc {
  TileShape shape;
  int S;
  // z tiles of runtime plans: rows, and 1 / (rows of a stage-0 block) where those
  // are padded apart (else 0)
  int zrows;
  float zpad;
  GenStage st[kBatchStages + 1];
};
template <typename T> struct alignas(16) GridHead {
  PassArgs<T> a;
  T *density;
  T *potential;
  int box_rows[2];   // rows per TMA box: y pass, x pass
};
template <typename T> struct alignas(16) GridDesc {
  GridHead<T> h;
  KindDesc k[5];
};

// ------------------------------------------------------------ column tiles
// A strided pass over W columns of the flattened column index
// q = plane * nhp + kh (FP64: nhp = nh): y columns are (i, kh) with rows j at
// stride nhp, x columns are (j, kh) with rows i at stride nj*nhp.  Consecutive q
// of one plane are contiguous, so every row access of a warp is coalesced.  FP32
// columns go in pairs (16 bytes); a row's padding column, if it has one, is
// transformed like the others and written back to the padding.  The tile
// arrives by asynchronous 16-byte copies (every load of the tile in flight at
// once: against loading stage 0 from HBM into registers FP64 batch x pass 0.87
// -> 0.68 ms, y 0.50 -> 0.44 ms), the stages run in the point-major tile, and
// the last stage writes HBM; all reads of a column precede the first barrier, so
// src may equal dst.  The x pass runs forward DIF, the -1/k^2 filter fused with
// the last DIF and first DIT stages, and the inverse DIT.  A thread owns one
// unit of 16 bytes in every stage (units fastest, the unit count divides the
// block).
template <typename T> struct ColsAt {
  using C = typename Cplx<T>::type;
  int o, kh;      // plane and first column of the unit
  long cb, rs;    // its first element and the row stride
  bool valid;
};
template <typename T, bool XPASS>
__device__ __forceinline__ ColsAt<T> cols_at(const PassArgs<T> &a, int tile, int W) {
  constexpr int CU = 16 / (2 * (int)sizeof(T));
  ColsAt<T> u;
  u.rs = XPASS ? (long)a.nj * a.nhp : (long)a.nhp;
  const long ps = XPASS ? (long)a.nhp : (long)a.nj * a.nhp;
  const int planes = XPASS ? a.nj : a.ni;
  const unsigned q = (unsigned)tile * W + CU * (threadIdx.x % (W / CU));
  u.valid = q < (unsigned)planes * a.nhp;
  u.o = u.valid ? (int)(q / (unsigned)a.nhp) : 0;
  u.kh = u.valid ? (int)(q - (unsigned)u.o * a.nhp) : 0;
  u.cb = (long)u.o * ps + u.kh;
  return u;
}
// The thread's units of n rows into the tile (rows of `units` units).
template <typename T, typename V>
__device__ __forceinline__ void cols_in(const ColsAt<T> &u, const typename Cplx<T>::type *src, V *sm, int n, int units) {
  const int c = threadIdx.x % units;
  for (int pos = threadIdx.x / units; pos < n; pos += kZThreads / units) {
    V *d = sm + pos * units + c;
    if (u.valid) cp_async16(d, src + u.cb + (long)pos * u.rs);
    else *reinterpret_cast<float4 *>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  cp_async_wait_all();
  __syncthreads();
}

// Stores of a column tile's last stage: row at(pos) of the thread's unit (FP32:
// pairs of columns).
template <typename C, typename RL> struct ColsStore {
  C *base;        // the unit's first element
  long rs;
  bool valid;
  RL rl;
  static constexpr bool kPair = std::is_same<C, float2>::value;
  __device__ __forceinline__ void operator()(int pos, int, C v) const {
    if (valid) base[(long)rl(pos) * rs] = v;
  }
  __device__ __forceinline__ void st2(int pos, int, float4 q) const {
    if (valid) *reinterpret_cast<float4 *>(base + (long)rl(pos) * rs) = q;
  }
};
struct SamePos {
  __device__ __forceinline__ int operator()(int pos) const { return pos; }
};

// Compile-time plans.
template <typename T, int W, bool XPASS, bool INV, int N>
__device__ __forceinline__ void cols_tile(const PassArgs<T> &a, const typename Cplx<T>::type *src,
                                          typename Cplx<T>::type *dst, int tile, typename Cplx<T>::type *sm) {
  using C = typename Cplx<T>::type;
  constexpr int NT = kZThreads;
  constexpr int CU = 16 / (int)sizeof(C);
  static_assert(NT % (W / CU) == 0, "a thread keeps one unit");
  const AxisDev<C> &ax = XPASS ? a.ax[0] : a.ax[1];
  const ColsAt<T> u = cols_at<T, XPASS>(a, tile, W);
  PointTile<W, C> tl{sm};
  cols_in(u, src, reinterpret_cast<float4 *>(sm), N, W / CU);
  // FP64 twiddle powers by recurrence, FP32 by table loads (as the single-grid passes)
  constexpr bool TWR = sizeof(T) == 8;
  if constexpr (!XPASS) {
    ColsStore<C, RevCT<N>> gst{dst + u.cb, u.rs, u.valid, RevCT<N>{}};
    dif_all<N, INV, Map::ColFast, W, NT, false, TWR>(ax, tl, tl, gst, W);
  } else {
    ColsStore<C, SamePos> gst{dst + u.cb, u.rs, u.valid, SamePos{}};
    // the filter's columns as one plane's: kh0 + c is the unit's column
    const double jd = double(min(u.o, a.nj - u.o)) * a.dd[1];
    const int c0 = CU * (int)(threadIdx.x % (W / CU));
    const XFilter flt{a.ni, u.o, u.kh - c0, u.valid ? W : 0, jd * jd, a.dd[0], a.dd[2], -a.invN};
    auto k0_of = [](int base) { return rev_ct<N>(base); };
    constexpr int S = plan_stages(N);
    constexpr int RF = plan_radix(N, S - 1);
    static_assert(S > 1, "the column tiles' lengths have two stages or more");
    dif_ct<N, S - 1, 0, false, Map::ColFast, W, NT, false, TWR>(ax, tl, tl, tl, W);
    x_filter_stage<RF, W, NT, N, C>(N, tl, tl, flt, k0_of, N / RF);
    __syncthreads();
    dit_ct<N, S - 2, true, Map::ColFast, W, NT, TWR>(ax, tl, gst, W);
  }
}

// Runtime plans (stages of ff_gen_stages.cuh in the radix order of the axis):
// a tile of the flattened columns, or (map) one plane's columns by TMA boxes.
// These and the z tiles below replace stages whose index work was four fifths of
// their instructions (222 warp instructions per 32 points of a y pass): 48 grids
// of ragged lengths FP64, z / y / x / y / z 252 / 203 / 297 / 205 / 268 -> 188 /
// 160 / 219 / 160 / 186 us.
template <typename T, bool XPASS, bool INV>
__device__ __forceinline__ bool cols_tile_rt(const PassArgs<T> &a, const GenStage *st, int S, int W,
                                             const typename Cplx<T>::type *src, typename Cplx<T>::type *dst,
                                             const CUtensorMap *map, int box_rows, int tile,
                                             typename Cplx<T>::type *sm, uint64_t *mbar, uint32_t &parity) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / (int)sizeof(C);
  const AxisDev<C> &ax = XPASS ? a.ax[0] : a.ax[1];
  const int units = W / CU, lu = 31 - __clz(units);
  V *tl = reinterpret_cast<V *>(sm);
  ColsAt<T> u;
  if (map) {
    constexpr int W1 = 128 / (int)sizeof(C);
    const int ktiles = (a.nh + W1 - 1) / W1;
    const int o = tile / ktiles, kt = tile - o * ktiles;
    if (!tma_tile<C, W1, XPASS>(map, sm, mbar, parity, ax.n, box_rows, o, kt, a.status)) return false;
    parity ^= 1u;
    u.o = o;
    u.kh = kt * W1 + CU * (int)(threadIdx.x % units);
    u.rs = XPASS ? (long)a.nj * a.nhp : (long)a.nhp;
    u.cb = (XPASS ? (long)o * a.nhp : (long)o * a.nj * a.nhp) + u.kh;
    u.valid = u.kh < a.nh;
  } else {
    u = cols_at<T, XPASS>(a, tile, W);
    cols_in(u, src, tl, ax.n, units);
  }
  const GenLane ln{(int)threadIdx.x & (units - 1), (int)threadIdx.x >> lu, kZThreads >> lu};
  const TileLoad<V> ld{tl, lu, ln.c};
  const TilePut<V> put{tl, lu, ln.c};
  const AxisTw<C> tw{ax.tw};
  using WAY = GenWay<false, 0>;
  gen_dif<WAY, XPASS ? false : INV>(st, S - 1, tw, ln, tl, lu, ld);
  const GenStage &s = st[S - 1];
  C *base = dst + u.cb;
  if constexpr (!XPASS) {
    with_gen_radix(s.R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      const long rs = (long)s.nb * u.rs;   // frequencies of a group are n/R apart
      for (int b = ln.b0; b < s.nb; b += ln.step) {
        const int k0 = __ldg(ax.rev + b * R);
        V v[R];
        ld.at(b * R, 1, v, tag);
        UDft<R, INV, V>::run(v);
        C *p = base + (long)k0 * u.rs;
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (u.valid) *reinterpret_cast<V *>(p) = v[r];
          p += rs;
        }
      }
    });
  } else {
    const double jd = double(min(u.o, a.nj - u.o)) * a.dd[1];
    const double ka = double(u.kh) * a.dd[2], kb = double(u.kh + 1) * a.dd[2];
    const GenFilter flt{a.ni, u.o, u.kh, jd * jd, a.dd[0], -a.invN, ka * ka, kb * kb};
    auto out = [&](int, int pos0, const GenStage &g, const V *v, auto tag) {
      C *p = base + (long)pos0 * u.rs;
      const long rs = (long)g.m * u.rs;
#pragma unroll
      for (int r = 0; r < decltype(tag)::value; r++) {
        if (u.valid) *reinterpret_cast<V *>(p) = v[r];
        p += rs;
      }
    };
    with_gen_radix(s.R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      for (int b = ln.b0; b < s.nb; b += ln.step) {
        const int k0 = __ldg(ax.rev + b * R);
        V v[R];
        ld.at(b * R, 1, v, tag);
        UDft<R, false, V>::run(v);
#pragma unroll
        for (int r = 0; r < R; r++) flt.apply(k0 + r * s.nb, v[r]);
        UDft<R, true, V>::run(v);
        if (S == 1) out(0, b * R, s, v, tag);
        else put(b * R, 0, s, v, tag);
      }
    });
    __syncthreads();
    for (int q = S - 2; q >= 0; q--) {
      with_gen_radix(st[q].R, [&](auto tag) {
        constexpr int R = decltype(tag)::value;
        if (q > 0) gen_stage<WAY, R, true, true, V>(st[q], tw, ln, ld, put);
        else gen_stage<WAY, R, true, true, V>(st[0], tw, ln, ld, out);
      });
      __syncthreads();
    }
  }
  return true;
}

// z tile of W line pairs of a runtime plan (ff_gen_lines.cuh).  bulk: the real
// lines move by one bulk copy (16-byte multiples), else by the threads; the
// spectrum rows always move by one copy.
template <typename T, bool INV>
__device__ __forceinline__ bool line_tile_rt(const PassArgs<T> &a, const KindDesc &k, const T *f, T *out,
                                             typename Cplx<T>::type *spec, bool bulk, int tile, unsigned char *sm,
                                             uint64_t *mbar, uint32_t &parity) {
  using C = typename Cplx<T>::type;
  const int nk = a.nk;
  const LineTileOf<C> b = line_tile<C>(nk, a.nhp, (long)a.ni * a.nj, k.shape.W, k.zrows, tile, sm);
  const ZTileIO io{mbar, parity, a.status};
  if (INV || bulk) {
    const bool ok = INV ? bulk_in(b.rows, spec + b.line0 * a.nhp, (size_t)b.nl * a.nhp * sizeof(C), io)
                        : bulk_in(b.raw, f + b.line0 * nk, (size_t)b.nl * nk * sizeof(T), io);
    parity ^= 1u;
    if (!ok) return false;
  } else {
    const T *src = f + b.line0 * nk;
    const int count = b.nl * nk;
    for (int q = threadIdx.x; q < count; q += blockDim.x) {
      if constexpr (sizeof(T) == 8) cp_async8(b.raw + q, src + q);
      else cp_async4(b.raw + q, src + q);
    }
    cp_async_wait_all();
    __syncthreads();
  }
  const AxisDev<C> &ax = a.ax[2];
  const AxisTw<C> tw{ax.tw};
  const float pad = k.zpad;
  auto row_of = [&](int k0) {
    const int pos = __ldg(ax.ipos + k0);
    return pos + __float2int_rz(((float)pos + 0.5f) * pad);
  };
  if constexpr (!INV) line_forward(b, k.st, k.S, tw, row_of);
  else line_inverse(b, k.st, k.S, tw, row_of);
  fence_proxy_async_smem();
  __syncthreads();
  if constexpr (!INV) {
    bulk_out(spec + b.line0 * a.nhp, b.rows, (size_t)b.nl * a.nhp);
  } else if (bulk) {
    bulk_out(out + b.line0 * nk, b.raw, (size_t)b.nl * nk);
  } else {
    T *dst = out + b.line0 * nk;
    for (int q = threadIdx.x; q < b.nl * nk; q += blockDim.x) dst[q] = b.raw[q];
  }
  return true;
}

// Strided tile with the column count chosen at run time: W * sizeof(C) is
// 128 * wb bytes.  Shapes whose tile exceeds the block budget are never
// planned and not instantiated.
template <typename T, bool XPASS, bool INV, int N>
__device__ __forceinline__ void cols_tile_w(int wb, const PassArgs<T> &a, const typename Cplx<T>::type *src,
                                            typename Cplx<T>::type *dst, int tile, typename Cplx<T>::type *sm) {
  using C = typename Cplx<T>::type;
  constexpr int W1 = 128 / (int)sizeof(C);
  constexpr bool fit2 = (size_t)N * 256 + 128 <= kBatchSmem;
  constexpr bool fit4 = (size_t)N * 512 + 128 <= kBatchSmem;
  if (wb == 4) {
    if constexpr (fit4) cols_tile<T, 4 * W1, XPASS, INV, N>(a, src, dst, tile, sm);
  } else if (wb == 2) {
    if constexpr (fit2) cols_tile<T, 2 * W1, XPASS, INV, N>(a, src, dst, tile, sm);
  } else {
    cols_tile<T, W1, XPASS, INV, N>(a, src, dst, tile, sm);
  }
}

// One tile of pass KIND of grid descriptor g.  Returns false if a bounded
// wait gave up (the status word is set).  parity tracks the block's
// mbarrier phase across the inbound bulk copies of the z inverse tiles.
// Strided tile of one plane by TMA (the single-grid tile code): W = 128
// bytes of kh columns, all n rows; tile = plane * ktiles + kt.
template <typename T, bool XPASS, bool INV, int N>
__device__ __forceinline__ bool tma_cols_tile(const GridHead<T> &g, const CUtensorMap *map, int tile,
                                              typename Cplx<T>::type *sm, uint64_t *mbar, uint32_t &parity) {
  using C = typename Cplx<T>::type;
  constexpr int W = 128 / (int)sizeof(C);
  const PassArgs<T> &a = g.a;
  const int n = XPASS ? a.ni : a.nj;
  const int ktiles = (a.nh + W - 1) / W;
  const int o = tile / ktiles, kt = tile - o * ktiles;
  const int box_rows = g.box_rows[XPASS ? 1 : 0];
  if (!tma_tile<C, W, XPASS>(map, sm, mbar, parity, n, box_rows, o, kt, a.status)) return false;
  parity ^= 1u;
  if constexpr (XPASS) {
    x_tile<T, W, N>(map, a, o, kt, box_rows, sm);
  } else {
    PointTile<W, C> t{sm};
    y_tile<T, W, INV, N>(t, reinterpret_cast<C *>(INV ? g.density : g.potential), a, o, kt, sm);
  }
  return true;
}

template <typename T, int KIND>
__device__ __forceinline__ bool batch_tile(const GridHead<T> &g, const KindDesc &k, const CUtensorMap *maps, int tile,
                                           typename Cplx<T>::type *sm, uint64_t *mbar, uint32_t &parity) {
  using C = typename Cplx<T>::type;
  const PassArgs<T> &a = g.a;
  const TileShape sh = k.shape;
  if constexpr (KIND == 0 || KIND == 4) {
    const int zW = sh.W;
    const int align = sizeof(C) == 16 ? 8 : 16;
    const int P = (a.nk + align - 1) / align * align;
    const long nlines = (long)a.ni * a.nj;
    const long line0 = (long)tile * 2 * zW;
    const ZTileIO io{mbar, parity, a.status};
    if constexpr (KIND == 0) {
      C *spec = reinterpret_cast<C *>(g.potential);
      if (sh.ct) {
        switch (a.nk) {
#define FF_CASE(NN) \
  case NN: {                                                                              \
    const bool ok = z_fwd_tile<T, NN, true, kBatchZThreads>(g.density, spec, a, zW, P, line0, nlines, sm, io); \
    parity ^= 1u;                                                                         \
    return ok;                                                                            \
  }
          FF_FOR_EACH_BATCH_N(FF_CASE)
#undef FF_CASE
          default: break;
        }
      }
      return line_tile_rt<T, false>(a, k, g.density, nullptr, spec, sh.tma != 0, tile,
                                    reinterpret_cast<unsigned char *>(sm), mbar, parity);
    } else {
      const C *spec = reinterpret_cast<const C *>(g.density);
      if (sh.ct) {
        switch (a.nk) {
#define FF_CASE(NN)                                                                       \
  case NN: {                                                                              \
    const bool ok = z_inv_tile<T, NN, true, kBatchZThreads>(spec, g.potential, a, zW, P, line0, nlines, sm, io); \
    parity ^= 1u;                                                                         \
    return ok;                                                                            \
  }
          FF_FOR_EACH_BATCH_N(FF_CASE)
#undef FF_CASE
          default: break;
        }
      }
      return line_tile_rt<T, true>(a, k, nullptr, g.potential, reinterpret_cast<C *>(g.density), sh.tma != 0, tile,
                                   reinterpret_cast<unsigned char *>(sm), mbar, parity);
    }
  } else {
    constexpr bool XPASS = KIND == 2;
    constexpr bool INV = KIND == 3;
    const C *src = reinterpret_cast<const C *>(g.potential);
    C *dst = reinterpret_cast<C *>(KIND == 3 ? g.density : g.potential);
    const int wb = sh.W * (int)sizeof(C) / 128;
    const int n = XPASS ? a.ni : a.nj;
    if (sh.tma) {
      const CUtensorMap *map = maps + (XPASS ? 1 : 0);
      // the grid's maps live in global memory and are rewritten when a
      // server slot changes hands
      if (threadIdx.x == 0) tensormap_acquire(map);
      if (sh.ct) {
        switch (n) {
#define FF_CASE(NN) \
  case NN: return tma_cols_tile<T, XPASS, INV, NN>(g, map, tile, sm, mbar, parity);
          FF_FOR_EACH_BATCH_TMA_N(FF_CASE)
#undef FF_CASE
          default: break;
        }
      }
      return cols_tile_rt<T, XPASS, INV>(a, k.st, k.S, sh.W, src, dst, map, g.box_rows[XPASS ? 1 : 0],
                                         tile, sm, mbar, parity);
    }
    if (sh.ct) {
      switch (n) {
#define FF_CASE(NN) \
  case NN: cols_tile_w<T, XPASS, INV, NN>(wb, a, src, dst, tile, sm); return true;
        FF_FOR_EACH_BATCH_N(FF_CASE)
#undef FF_CASE
        default: break;
      }
    }
    return cols_tile_rt<T, XPASS, INV>(a, k.st, k.S, sh.W, src, dst, nullptr, 0, tile, sm, mbar, parity);
  }
}

// The entry of tile t: the largest e with start[e] <= t, by every warp for itself,
// 32 entries a step; *base = start[e].
__device__ __forceinline__ int batch_entry(const int *__restrict__ start, int count, int t, int *base) {
  const int lane = threadIdx.x & 31;
  int lo = 0, first = 0;
  for (int left = count; left > 0;) {
    const int step = (left + 31) >> 5;
    const bool in = lane * step < left;
    const int v = in ? __ldg(start + lo + lane * step) : 0;
    const int k = 31 - __clz(__ballot_sync(0xffffffffu, in && v <= t));   // start[lo] <= t throughout
    first = __shfl_sync(0xffffffffu, v, k);
    lo += k * step;
    left = step > 1 ? min(step, left - k * step) : 0;
  }
  *base = first;
  return lo;
}

// Pass kernel: one tile per block, in the order of the work list.  (Persistent
// blocks that took tiles from a counter spent a round trip of the atomic, the
// search and the descriptor read between a tile's last store and the next one's
// first load; the hardware starts the next block's while other blocks still work.
// 60 grids of 32 to 128 points FP32: 497 -> 457 us a batch; 48 grids of ragged
// lengths up to 160 FP64: 1017 -> 916.)
template <typename T, int KIND>
__global__ void __launch_bounds__((KIND == 0 || KIND == 4) ? kBatchZThreads : kZThreads,
                                  (KIND == 0 || KIND == 4) ? 6 : 3)
    k_batch(const GridDesc<T> *__restrict__ grids, const CUtensorMap *__restrict__ maps, const BatchWork wl) {
  using C = typename Cplx<T>::type;
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ GridHead<T> s_head;
  __shared__ KindDesc s_kind;
  C *sm = reinterpret_cast<C *>(align128(smraw));
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_init_fence();
  }
  const int t = blockIdx.x;
  int first = 0;
  const int g = wl.entry[batch_entry(wl.start, wl.nentry, t, &first)];
  {
    // descriptor of the tile's grid into shared memory (read-only below)
    constexpr int kHead = sizeof(GridHead<T>) / 16, kKind = sizeof(KindDesc) / 16;
    const int4 *sh = reinterpret_cast<const int4 *>(&grids[g].h), *sk = reinterpret_cast<const int4 *>(&grids[g].k[KIND]);
    int4 *dh = reinterpret_cast<int4 *>(&s_head), *dk = reinterpret_cast<int4 *>(&s_kind);
    for (int w = threadIdx.x; w < kHead + kKind; w += blockDim.x) {
      if (w < kHead) dh[w] = __ldg(sh + w);
      else dk[w - kHead] = __ldg(sk + (w - kHead));
    }
  }
  if constexpr (KIND == 0 || KIND == 4) {
    // z passes: the last warp hints the input of the tile one resident wave
    // ahead into L2
    const int t2 = t + wl.ahead;
    int first2 = 0;
    if (threadIdx.x >= kBatchZThreads - 32 && t2 < (int)gridDim.x) {
      const GridDesc<T> *G = grids + wl.entry[batch_entry(wl.start, wl.nentry, t2, &first2)];
      if (threadIdx.x == kBatchZThreads - 32) {
        const int zW = G->k[KIND].shape.W;
        const long nlines = (long)G->h.a.ni * G->h.a.nj;
        // real lines, within the buffer (max(real field, half spectrum) bytes), or
        // spectrum rows
        const size_t spec = (size_t)G->h.a.nhp * 2 * sizeof(T);
        const size_t row = KIND == 0 ? (size_t)G->h.a.nk * sizeof(T) : spec;
        const size_t cap = nlines * (row > spec ? row : spec);
        const long l0 = (long)(t2 - first2) * 2 * zW;
        const long l1 = min(l0 + 2 * zW, nlines);
        const size_t b0 = (l0 * row) & ~size_t(15);
        const size_t b1 = min((l1 * row + 15) & ~size_t(15), cap & ~size_t(15));
        l2_prefetch(reinterpret_cast<const char *>(G->h.density) + b0, (uint32_t)(b1 - b0));
      }
    }
  }
  __syncthreads();
  uint32_t parity = 0;
  batch_tile<T, KIND>(s_head, s_kind, maps + 2 * g, t - first, sm, &mbar, parity);
}

template <typename T, int KIND> static void *batch_kernel_ptr() { return (void *)k_batch<T, KIND>; }

template <typename T> static void *batch_kernel(int kind) {
  switch (kind) {
    case 0: return batch_kernel_ptr<T, 0>();
    case 1: return batch_kernel_ptr<T, 1>();
    case 2: return batch_kernel_ptr<T, 2>();
    case 3: return batch_kernel_ptr<T, 3>();
    default: return batch_kernel_ptr<T, 4>();
  }
}

template <typename T>
int batch_pass_launch(int kind, const void *grids, const CUtensorMap *maps, const BatchWork &wl, int blocks,
                      size_t smem, cudaStream_t st) {
  const GridDesc<T> *g = static_cast<const GridDesc<T> *>(grids);
  switch (kind) {
    case 0: k_batch<T, 0><<<blocks, batch_threads(0), smem, st>>>(g, maps, wl); break;
    case 1: k_batch<T, 1><<<blocks, batch_threads(1), smem, st>>>(g, maps, wl); break;
    case 2: k_batch<T, 2><<<blocks, batch_threads(2), smem, st>>>(g, maps, wl); break;
    case 3: k_batch<T, 3><<<blocks, batch_threads(3), smem, st>>>(g, maps, wl); break;
    default: k_batch<T, 4><<<blocks, batch_threads(4), smem, st>>>(g, maps, wl); break;
  }
  FF_CUDA(cudaGetLastError());
  return FF_OK;
}

template <typename T> int batch_pass_prepare(int kind, size_t smem, int *per_sm) {
  const void *fn = batch_kernel<T>(kind);
  cudaFuncAttributes fa;
  FF_CUDA(cudaFuncGetAttributes(&fa, fn));
  if (fa.sharedSizeBytes + batch_budget(kind) > 227 * 1024)
    return set_error(FF_ERR_UNSUPPORTED, "batch kernel shared memory exceeds the block limit");
  FF_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)batch_budget(kind)));
  FF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, fn, batch_threads(kind), smem));
  return FF_OK;
}

template <typename T> size_t batch_desc_size() { return sizeof(GridDesc<T>); }

template <typename T> void batch_desc_fill(void *dst, const BatchGridHost &h) {
  GridDesc<T> d;
  memset(&d, 0, sizeof(d));
  GridHead<T> &g = d.h;
  g.a.ni = h.n[0];
  g.a.nj = h.n[1];
  g.a.nk = h.n[2];
  g.a.nh = h.nh;
  g.a.nhp = h.nhp;
  for (int d = 0; d < 3; d++) {
    if constexpr (sizeof(T) == 8) g.a.ax[d] = h.axd[d];
    else g.a.ax[d] = h.axf[d];
    g.a.dd[d] = h.dd[d];
  }
  g.a.invN = h.invN;
  g.a.status = h.status;
  g.a.l2_ahead = 0;
  g.density = static_cast<T *>(h.density);
  g.potential = static_cast<T *>(h.potential);
  g.box_rows[0] = h.box_rows[0];
  g.box_rows[1] = h.box_rows[1];
  for (int k = 0; k < 5; k++) {
    KindDesc &kd = d.k[k];
    kd.shape = h.shape[k];
    const int axis = k == 0 || k == 4 ? 2 : k == 2 ? 0 : 1;
    const AxisDev<double2> &ax = h.axd[axis];
    const std::vector<int> radix(ax.radix, ax.radix + ax.nstages);
    if (axis == 2) {
      const int pad = gen_pad(ax.n, radix);
      kd.zrows = ax.n + pad * (radix[0] - 1);
      kd.zpad = pad ? (float)radix[0] / (float)ax.n : 0.0f;
      gen_line_stages(ax.n, radix, pad, batch_threads(k), true, &kd.S, kd.st);
    } else {
      const int units = h.shape[k].W * 2 * (int)sizeof(T) / 16;
      gen_stages(ax.n, radix, 0, batch_threads(k), units, &kd.S, kd.st);
      for (int s = 0, step = 1; s < kd.S; s++) {
        kd.st[s].tw = step;   // the plain table's step
        step *= kd.st[s].R;
      }
    }
  }
  memcpy(dst, &d, sizeof(d));
}

#define FF_INSTANTIATE_BATCH(T)                                                                               \
  template int batch_pass_launch<T>(int, const void *, const CUtensorMap *, const BatchWork &, int, size_t,   \
                                    cudaStream_t);                                                          \
  template int batch_pass_prepare<T>(int, size_t, int *);                                                    \
  template size_t batch_desc_size<T>();                                                                      \
  template void batch_desc_fill<T>(void *, const BatchGridHost &);

}  // namespace ff
