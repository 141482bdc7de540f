// Kernels of the passes along axes without a compile-time plan.  Included by
// ff_gen_f64.cu and ff_gen_f32.cu, one precision each.
//
// The stages are those of ff_gen_stages.cuh.
//
// A plan read at run time costs integer work: a digit reversal with a remainder
// for each output, a quotient for each butterfly and five-factor plans took
// 338 (z) and 180 (y) warp instructions per 32 complex points at 480x400x360 FP64, a
// fifth of them FP64.  So here
//   - radices go up to 10 (6 and 10 without inner twiddles, by the prime factor
//     algorithm), which makes three stages of nearly every length up to 1000;
//   - the butterfly's block and offset advance by additions;
//   - a butterfly's points are one pointer and a uniform stride on both sides
//     (the last stage of a forward transform has frequencies k0 + r n/R, so its
//     stores to HBM or to staged rows are one too): one table load per group;
//   - twiddles lie per stage as [j][r], one address for a butterfly's factors;
//   - the z passes fuse the last stage with the real split as the compile-time
//     ones do, in one form for every radix.
// One B200, passes z / y / x / y / z with and without all that: 480x400x360 FP64
// 483 / 328 / 424 / 326 / 581 us -> 236 / 222 / 345 / 214 / 241 (2.14 -> 1.26 ms a
// solve, 68 % of the copy rate over the five passes' bytes); FP32 332 / 229 / 301 /
// 232 / 369 -> 137 / 137 / 205 / 136 / 144 (1.46 -> 0.76 ms).
//
// What bounds them: no pipe is saturated (480x400x360 FP64 y pass: DRAM 60 %,
// L1 55 %, FP64 32 %, issue 37 %); a block's load, its stages and its stores
// follow one another, and 24 warps on an SM (80 registers) overlap them across
// blocks.  Persistent blocks with two tile buffers, so that no warp waits for a
// load, need blocks of twice the size, half as many: their warps then load, add
// and store in step, which cost more than it hid (y 217 -> 290, x 335 -> 417,
// z 245 -> 350 us).  64 registers and 32 warps spill (y 217 -> 247 us).
#pragma once

#include "ff_gen_lines.cuh"
#include "ff_launch.hpp"

namespace ff {

// --------------------------------------------------------- strided passes
// One TMA-filled tile per block: units * 16 bytes of kh columns by all n rows
// of one plane.  y: the last stage stores straight to HBM; x: last forward
// stage, filter and first inverse stage on one register group, then back into
// the tile and out by TMA.
template <bool INV, typename C, typename V>
__device__ __forceinline__ void gen_y_last(const GenPass<C> &a, const GenLane &ln, const V *tile, C *plane, int col0) {
  const GenStage &s = a.ax.st[a.ax.S - 1];
  const TileLoad<V> ld{tile, a.lu, ln.c};
  constexpr int CU = 16 / sizeof(C);   // columns per unit
  const int col = col0 + ln.c * CU;
  if (col >= a.nh) return;
  const bool whole = CU == 1 || col + 1 < a.nh;
  const long rs = (long)s.nb * a.nhp;   // frequencies of a group are n/R apart
  with_gen_radix(s.R, [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    for (int b = ln.b0; b < s.nb; b += ln.step) {
      const int k0 = __ldg(a.ax.idx + b);
      V v[R];
      ld.at(b * R, 1, v, tag);
      UDft<R, INV, V>::run(v);
      C *p = plane + (long)k0 * a.nhp + col;
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (whole) *reinterpret_cast<V *>(p) = v[r];
        else if constexpr (CU == 2) *p = v[r].a;
        p += rs;
      }
    }
  });
}

template <typename C, typename V>
__device__ __forceinline__ void gen_x_tile(const GenPass<C> &a, const GenLane &ln, V *tile, int j, int col0) {
  const int S = a.ax.S;
  const TileLoad<V> ld{tile, a.lu, ln.c};
  const TilePut<V> put{tile, a.lu, ln.c};
  gen_dif<GenStrided<C>, false>(a.ax.st, S - 1, PackedTw<C>{a.ax.tw}, ln, tile, a.lu, ld);
  {
    constexpr int CU = 16 / sizeof(C);
    const GenStage &s = a.ax.st[S - 1];
    const double jd = double(min(j, a.nj - j)) * a.dd[1];
    const int kh = col0 + ln.c * CU;
    const double ka = double(kh) * a.dd[2], kb = double(kh + 1) * a.dd[2];
    const GenFilter flt{a.ni, j, kh, jd * jd, a.dd[0], -a.invN, ka * ka, kb * kb};
    with_gen_radix(s.R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      for (int b = ln.b0; b < s.nb; b += ln.step) {
        const int k0 = __ldg(a.ax.idx + b);
        V v[R];
        ld.at(b * R, 1, v, tag);
        UDft<R, false, V>::run(v);
        // columns past nh hold what the tensor map fills in (zero)
#pragma unroll
        for (int r = 0; r < R; r++) flt.apply(k0 + r * s.nb, v[r]);
        UDft<R, true, V>::run(v);
        V *p = tile + ((b * R) << a.lu) + ln.c;
#pragma unroll
        for (int r = 0; r < R; r++) p[r << a.lu] = v[r];
      }
    });
    __syncthreads();
  }
  for (int s = S - 2; s >= 0; s--) {
    with_gen_radix(a.ax.st[s].R, [&](auto tag) {
      gen_stage<GenStrided<C>, decltype(tag)::value, true, true, V>(a.ax.st[s], PackedTw<C>{a.ax.tw}, ln, ld, put);
    });
    __syncthreads();
  }
}

// KIND 1: y forward, 2: x, 3: y inverse.
template <typename T, int KIND>
__global__ void __launch_bounds__(256, 3)
    k_gen_strided(const __grid_constant__ CUtensorMap tmap, typename Cplx<T>::type *dst,
                  const __grid_constant__ GenPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr bool XPASS = KIND == 2;
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  V *tile = reinterpret_cast<V *>(align128(smraw));
  const int n = a.ax.n;
  const int W = (16 / (int)sizeof(C)) << a.lu;
  const int ktiles = (a.nh + W - 1) / W;
  const int o = blockIdx.x / ktiles, kt = blockIdx.x - o * ktiles;
  const int rows = a.box_rows;
  pdl_start();
  pdl_wait();
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_init_fence();
    mbar_expect_tx(&mbar, (uint32_t)((n + rows - 1) / rows * rows << a.lu) * 16);
    for (int q = 0; q < n; q += rows) {
      if (XPASS) tma_load_3d(tile + (q << a.lu), &tmap, 2 * W * kt, o, q, &mbar);
      else tma_load_3d(tile + (q << a.lu), &tmap, 2 * W * kt, q, o, &mbar);
    }
  }
  __syncthreads();
  const bool ok = mbar_wait_bounded(&mbar, 0, a.wait_iters);
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) {
      atomicExch(a.status, kDevTmaTimeout);
      mbar_wait_bounded(&mbar, 0);
    }
    return;
  }
  const GenLane ln = gen_lane(a);
  if constexpr (XPASS) {
    gen_x_tile(a, ln, tile, o, kt * W);
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int q = 0; q < n; q += rows) tma_store_3d(&tmap, 2 * W * kt, o, q, tile + (q << a.lu));
      bulk_commit();
      bulk_wait_read();
    }
  } else {
    const TileLoad<V> ld{tile, a.lu, ln.c};
    gen_dif<GenStrided<C>, KIND == 3>(a.ax.st, a.ax.S - 1, PackedTw<C>{a.ax.tw}, ln, tile, a.lu, ld);
    gen_y_last<KIND == 3>(a, ln, tile, dst + (long)o * a.nj * a.nhp, kt * W);
  }
}

// ------------------------------------------------------------- z passes
// A block holds `units` columns of line pairs: FP64 unit c is the pair of lines
// (2c, 2c+1); FP32 unit c holds that pair and the pair of lines (2u + 2c,
// 2u + 2c + 1), u the tile's units.  Two buffers: the tile and the staging area
// (real lines of pitch lp on one side, spectrum rows of pitch sp on the other).
// Lines at or past the end are zero in and not stored.
//
// FP32: z tiles with butterflies fastest (ff_gen_lines.cuh), whose unpadded
// staging moves by one copy each way: 480x400x360 z 162 / 160 -> 141 / 143 us,
// 640x640x320 306 / 296 -> 242 / 254.  (FP64 lost with them: 243 / 240 -> 250 /
// 260 and 480^3 368 / 349 -> 410 / 429, their last rows and twiddles being twice
// as wide; it keeps units fastest.)
template <int KIND>
__global__ void __launch_bounds__(256, 3)
    k_gen_lines(const void *in, void *out, const __grid_constant__ GenPass<float2> a) {
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const long nlines = (long)a.ni * a.nj;
  const LineTileOf<float2> b =
      line_tile<float2>(a.nk, a.nhp, nlines, 2 << a.lu, a.tile_rows, blockIdx.x, align128(smraw));
  // rows in and out, in bytes
  const size_t rin = KIND == 0 ? a.nk * sizeof(float) : a.nhp * sizeof(float2);
  const unsigned char *src = static_cast<const unsigned char *>(in);
  if (KIND == 0) pdl_start();
  pdl_wait();
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_init_fence();
    // one copy rounded up to 16 bytes: a real field's buffer also holds the
    // half spectrum, which is longer; spectrum rows are 16-byte multiples
    const uint32_t bytes = (uint32_t)(b.nl * rin + 15) & ~15u;
    mbar_expect_tx(&mbar, bytes);
    bulk_load(b.raw, src + b.line0 * rin, bytes, &mbar);
  }
  if (threadIdx.x == blockDim.x - 1 && a.l2_ahead > 0) {
    const long fl = b.line0 + (long)a.l2_ahead * b.lines;
    if (fl < nlines) l2_prefetch(src + fl * rin, (uint32_t)(min((long)b.lines, nlines - fl) * rin));
  }
  __syncthreads();
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  const PackedTw<float2> tw{a.ax.tw};
  auto row_of = [&](int k0) { return __ldg(a.ax.idx + k0); };
  if constexpr (KIND == 0) line_forward(b, a.ax.st, a.ax.S, tw, row_of);
  else line_inverse(b, a.ax.st, a.ax.S, tw, row_of);
  fence_proxy_async_smem();
  __syncthreads();
  if constexpr (KIND == 0) bulk_out(static_cast<float2 *>(out) + b.line0 * a.nhp, b.rows, (size_t)b.nl * a.nhp);
  else bulk_out(static_cast<float *>(out) + b.line0 * a.nk, b.raw, (size_t)b.nl * a.nk);
}

// R2C of the real lines (ParisPencil.cpp:152-165).
template <typename T>
__global__ void __launch_bounds__(256, 3)
    k_gen_zfwd(const T *__restrict__ f, typename Cplx<T>::type *spec,
               const __grid_constant__ GenPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  static_assert(sizeof(C) == 16, "FP32 takes k_gen_lines");
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const int nk = a.nk, units = 1 << a.lu, lines = 2 * units;
  V *tile = reinterpret_cast<V *>(align128(smraw));
  unsigned char *stage = reinterpret_cast<unsigned char *>(tile + ((((a.tile_rows << a.lu) + 7) >> 3) << 3));
  T *raw = reinterpret_cast<T *>(stage);
  const long nlines = (long)a.ni * a.nj;
  const long line0 = (long)blockIdx.x * lines;
  const int nl = (int)min((long)lines, nlines - line0);
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_init_fence();
  }
  pdl_start();
  pdl_wait();
  __syncthreads();
  lines_in(a, raw, f, line0, nl, &mbar);
  if (threadIdx.x == blockDim.x - 1 && a.l2_ahead > 0) {
    // the lines of the block one resident wave ahead into L2
    const long fl = ((long)blockIdx.x + a.l2_ahead) * lines;
    if (fl < nlines)
      l2_prefetch(f + fl * nk, (uint32_t)((size_t)min((long)lines, nlines - fl) * nk * sizeof(T)));
  }
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  if (nl < lines) {
    for (int q = nl * a.lp + threadIdx.x; q < lines * a.lp; q += blockDim.x) raw[q] = (T)0;
    __syncthreads();
  }
  const GenLane ln = gen_lane(a);
  const T *ra = raw + 2 * ln.c * a.lp;
  auto ld0 = [&](int, int pos, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
    const T *p = ra + pos;
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = unit_of<V>(p + r * st.m, a.lp, 0);
  };
  const int S = a.ax.S;
  if (S > 1) {
    gen_dif<GenLines, false>(a.ax.st, S - 1, PackedTw<C>{a.ax.tw}, ln, tile, a.lu, ld0);
  } else {
    // one stage: the split reads the tile
    for (int pos = ln.b0; pos < nk; pos += ln.step) ld0(pos, pos, a.ax.st[0], tile + (pos << a.lu) + ln.c, RadixTag<1>{});
    __syncthreads();
  }
  // Last stage and split: the groups of bases k0 and nR - k0 (nR = n/R) hold
  // Z[k0 + r nR] and, at R-1-r, Z[n - (k0 + r nR)]; base 0 pairs with itself
  // shifted by one and nR/2 with itself (their pairs come out twice, the same
  // values).  A[k] = (Z[k] + conj Z[n-k]) / 2 and B[k] = (Z[k] - conj Z[n-k]) /
  // (2i) go to the staged rows of the pair's lines.
  const GenStage &s = a.ax.st[S - 1];
  C *out = reinterpret_cast<C *>(stage) + 2 * ln.c * a.sp;
  const int nR = s.nb;
  const TileLoad<V> ld{tile, a.lu, ln.c};
  with_split_radix(s.R, [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    for (int k0 = ln.b0; 2 * k0 <= nR; k0 += ln.step) {
      V z1[R], z2[R];
      ld.at(__ldg(a.ax.idx + k0), 1, z1, tag);
      UDft<R, false, V>::run(z1);
      if (k0 > 0) {
        ld.at(__ldg(a.ax.idx + nR - k0), 1, z2, tag);
        UDft<R, false, V>::run(z2);
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) z2[r] = z1[(r + 1) % R];
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
        const bool low = 2 * r < R;
        const int k = low ? k0 + r * nR : nk - k0 - r * nR;
        const V p = low ? z1[r] : z2[R - 1 - r], q = low ? z2[R - 1 - r] : z1[r];   // Z[k], Z[n - k]
        unit_split(out + k, a.sp, 0, p, q);
      }
    }
  });
  fence_proxy_async_smem();
  __syncthreads();
  rows_out(reinterpret_cast<unsigned char *>(spec + line0 * a.nhp), a.nhp * sizeof(C), stage, a.sp * sizeof(C), nl);
}

// C2R of the spectrum rows (ParisPencil.cpp:368-380).
template <typename T>
__global__ void __launch_bounds__(256, 3)
    k_gen_zinv(const typename Cplx<T>::type *spec, T *__restrict__ f,
               const __grid_constant__ GenPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  static_assert(sizeof(C) == 16, "FP32 takes k_gen_lines");
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const int nk = a.nk, units = 1 << a.lu, lines = 2 * units;
  V *tile = reinterpret_cast<V *>(align128(smraw));
  unsigned char *stage = reinterpret_cast<unsigned char *>(tile + ((((a.tile_rows << a.lu) + 7) >> 3) << 3));
  C *rows = reinterpret_cast<C *>(stage);
  const long nlines = (long)a.ni * a.nj;
  const long line0 = (long)blockIdx.x * lines;
  const int nl = (int)min((long)lines, nlines - line0);
  if (threadIdx.x == 0) {
    mbar_init(&mbar, 1);
    mbar_init_fence();
  }
  pdl_wait();
  __syncthreads();
  rows_in(stage, a.sp * sizeof(C), reinterpret_cast<const unsigned char *>(spec + line0 * a.nhp), a.nhp * sizeof(C), nl,
          &mbar);
  if (threadIdx.x == blockDim.x - 1 && a.l2_ahead > 0) {
    const long fl = ((long)blockIdx.x + a.l2_ahead) * lines;
    if (fl < nlines)
      l2_prefetch(spec + fl * a.nhp, (uint32_t)((size_t)min((long)lines, nlines - fl) * a.nhp * sizeof(C)));
  }
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  z_rows_real_ends(a, rows, nl, lines);
  __syncthreads();
  const GenLane ln = gen_lane(a);
  const C *ra = rows + 2 * ln.c * a.sp;
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = unit_extend<V>(ra, a.sp, 0, nk, pos0 + r * st.m);
  };
  const int S = a.ax.S;
  if (S > 1) {
    gen_dif<GenLines, true>(a.ax.st, S - 1, PackedTw<C>{a.ax.tw}, ln, tile, a.lu, ld0);
  } else {
    for (int pos = ln.b0; pos < nk; pos += ln.step) ld0(pos, pos, a.ax.st[0], tile + (pos << a.lu) + ln.c, RadixTag<1>{});
    __syncthreads();
  }
  // last stage: real and imaginary parts of points k0 + r n/R to the two real
  // lines of the pair
  const GenStage &s = a.ax.st[S - 1];
  T *out = reinterpret_cast<T *>(stage) + 2 * ln.c * a.lp;
  const TileLoad<V> ld{tile, a.lu, ln.c};
  with_split_radix(s.R, [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    for (int k0 = ln.b0; k0 < s.nb; k0 += ln.step) {
      V z[R];
      ld.at(__ldg(a.ax.idx + k0), 1, z, tag);
      UDft<R, true, V>::run(z);
      T *o = out + k0;
#pragma unroll
      for (int r = 0; r < R; r++) {
        unit_put(o, a.lp, 0, z[r]);
        o += s.nb;
      }
    }
  });
  fence_proxy_async_smem();
  __syncthreads();
  if (a.per_line)
    rows_out(reinterpret_cast<unsigned char *>(f + line0 * nk), nk * sizeof(T), stage, a.lp * sizeof(T), nl);
  else
    bulk_out(f + line0 * nk, reinterpret_cast<const T *>(stage), (size_t)nl * nk);
}

// ----------------------------------------------------------------- launches
template <typename T> const void *gen_kernel(int kind) {
  switch (kind) {
    case 0:
      if constexpr (sizeof(T) == 4) return (const void *)k_gen_lines<0>;
      else return (const void *)k_gen_zfwd<T>;
    case 1: return (const void *)k_gen_strided<T, 1>;
    case 2: return (const void *)k_gen_strided<T, 2>;
    case 3: return (const void *)k_gen_strided<T, 3>;
    default:
      if constexpr (sizeof(T) == 4) return (const void *)k_gen_lines<4>;
      else return (const void *)k_gen_zinv<T>;
  }
}

int allow_dyn_smem_fn(const void *fn, size_t *avail);

template <typename T> int gen_prepare(int kind, size_t smem) {
  size_t avail = 0;
  const int rc = allow_dyn_smem_fn(gen_kernel<T>(kind), &avail);
  if (rc != FF_OK) return rc;
  if (smem > avail) return set_error(FF_ERR_UNSUPPORTED, "a tile of %zu bytes does not fit in shared memory", smem);
  return FF_OK;
}

template <typename T>
int gen_launch(int kind, const GenPass<typename Cplx<T>::type> &a, const GenShape &s, const CUtensorMap *map,
               const void *in, void *out, cudaStream_t st) {
  using C = typename Cplx<T>::type;
  auto go = [&](auto k, auto... args) { return launch_chained(s.chained, k, (unsigned)s.grid, s.threads, s.smem, st, args...); };
  cudaError_t e;
  switch (kind) {
    case 0:
      if constexpr (sizeof(T) == 4) e = go(k_gen_lines<0>, in, out, a);
      else e = go(k_gen_zfwd<T>, static_cast<const T *>(in), static_cast<C *>(out), a);
      break;
    case 1: e = go(k_gen_strided<T, 1>, *map, static_cast<C *>(out), a); break;
    case 2: e = go(k_gen_strided<T, 2>, *map, static_cast<C *>(out), a); break;
    case 3: e = go(k_gen_strided<T, 3>, *map, static_cast<C *>(out), a); break;
    default:
      if constexpr (sizeof(T) == 4) e = go(k_gen_lines<4>, in, out, a);
      else e = go(k_gen_zinv<T>, static_cast<const C *>(in), static_cast<T *>(out), a);
      break;
  }
  FF_CUDA(e);
  return FF_OK;
}

#define FF_INSTANTIATE_GEN(T)                                                                               \
  template int gen_prepare<T>(int, size_t);                                                                 \
  template int gen_launch<T>(int, const GenPass<typename Cplx<T>::type> &, const GenShape &, const CUtensorMap *, \
                             const void *, void *, cudaStream_t);

}  // namespace ff
