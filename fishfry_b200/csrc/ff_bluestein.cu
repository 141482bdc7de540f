// Bluestein passes of the single-grid solve for axes with a prime factor
// above 7 (the algorithm and its tables are described in ff_bluestein.hpp).
//
// One kernel per pass kind, on the stages of the generic passes (16-byte
// units, radices up to 10, plan read at run time):
//   z forward / inverse: `units` columns of line pairs per block; the lines
//     arrive in a staging area by bulk copies and the result leaves from it;
//   y forward / inverse, x: `units` spectrum columns x M rows per block, rows
//     read and written directly from HBM (the tile holds M > n rows, so it is
//     not the box a TMA copy would move).
// The x kernel runs the forward transform, stores the filtered spectrum in
// place through its last stage, and runs the inverse on the same tile.
//
// Each direction is two M-point transforms, M >= 2n - 1: the passes are bound by
// their stages (instruction issue and shared memory), not by HBM.  M is
// the cheapest smooth length, not the smallest (bs_padded_length).  One B200, passes z / y / x / y / z:
// 211^3 FP64 295 / 193 / 391 / 193 / 295 us on the earlier stages with one radix
// split for all M, 121 / 120 / 209 / 115 / 127 now; 256x256x251 FP64 z 387 / 387
// -> 255 / 259, FP32 266 / 275 -> 132 / 133.

#include <cuda_runtime.h>

#include <algorithm>

#include "ff_bluestein.hpp"
#include "ff_gen_stages.cuh"
#include "ff_launch.hpp"

namespace ff {

int allow_dyn_smem_fn(const void *fn, size_t *avail);
double gen_cost(int n);

namespace {

// The circular convolution of the tile's lines with the chirp kernel: stage 0
// reads ld0 (the premultiplied line, zero from n to M); the result leaves
// through put from the last inverse stage, in natural order: put(row, pos, s, v)
// has conv[pos + r m].  INV selects the conjugate kernel.  A block barrier follows.
template <typename WAY, bool INV, typename V, typename C, typename LD0, typename ST>
__device__ __forceinline__ void bs_conv(const BsPass<C> &a, const GenLane &ln, V *tile, LD0 &&ld0, ST &&put) {
  const GenAxis<C> &ax = a.ax;
  const int S = ax.S;   // n >= 11, so M >= 21: at least two stages
  const TileLoad<V> ld{tile, a.lu, ln.c};
  const TilePut<V> back{tile, a.lu, ln.c};
  gen_dif<WAY, false>(ax.st, S - 1, PackedTw<C>{ax.tw}, ln, tile, a.lu, ld0);
  with_gen_radix(ax.st[S - 1].R, [&](auto tag) {
    // the last DIF stage, the product with ghat and the first DIT stage on one
    // register group (the span-R stages have no twiddles)
    constexpr int R = decltype(tag)::value;
    const int nb = ax.st[S - 1].nb;
    for (int b = ln.b0; b < nb; b += ln.step) {
      V v[R];
      ld.at(b * R, 1, v, tag);
      UDft<R, false, V>::run(v);
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = ucmul<INV>(v[r], __ldg(a.ghat + b * R + r));
      UDft<R, true, V>::run(v);
      back(b * R, 0, ax.st[S - 1], v, tag);
    }
  });
  __syncthreads();
  for (int s = S - 2; s >= 0; s--) {
    with_gen_radix(ax.st[s].R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      if (s > 0) gen_stage<WAY, R, true, true, V>(ax.st[s], PackedTw<C>{ax.tw}, ln, ld, back);
      else gen_stage<WAY, R, true, true, V>(ax.st[0], PackedTw<C>{ax.tw}, ln, ld, put);
    });
    __syncthreads();
  }
}

using BsWay = GenWay<false, 0>;

__device__ __forceinline__ double2 zero_unit(double2 *) { return mk(0.0, 0.0); }
__device__ __forceinline__ FPair zero_unit(FPair *) { return {mk(0.0f, 0.0f), mk(0.0f, 0.0f)}; }

template <typename C> __device__ __forceinline__ GenLane bs_lane(const BsPass<C> &a) {
  return {(int)threadIdx.x & ((1 << a.lu) - 1), (int)threadIdx.x >> a.lu, (int)blockDim.x >> a.lu};
}

// R2C along z (ParisPencil.cpp:152-165).
template <typename T>
__global__ void __launch_bounds__(256, 3)
    k_bs_zfwd(const T *__restrict__ f, typename Cplx<T>::type *spec,
              const __grid_constant__ BsPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / sizeof(C);
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const int nk = a.nk, units = 1 << a.lu, lines = 2 * CU * units;
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
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  if (nl < lines) {
    for (int q = nl * a.lp + threadIdx.x; q < lines * a.lp; q += blockDim.x) raw[q] = (T)0;
    __syncthreads();
  }
  const GenLane ln = bs_lane(a);
  const T *ra = raw + 2 * ln.c * a.lp;
  const int second = 2 * units * a.lp;
  // two real lines as one complex line, times the chirp; zero from nk on
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if (pos < nk) {
        const T *q = ra + pos;
        if constexpr (CU == 1) v[r] = mk(q[0], q[a.lp]);
        else v[r] = {mk(q[0], q[a.lp]), mk(q[second], q[second + a.lp])};
        v[r] = ucmul<false>(v[r], __ldg(a.chirp + pos));
      } else {
        v[r] = zero_unit((V *)nullptr);
      }
    }
  };
  bs_conv<BsWay, false>(a, ln, tile, ld0, TilePut<V>{tile, a.lu, ln.c});
  // Z[k] = chirp[k] conv[k]; A[k] = (Z[k] + conj Z[n-k]) / 2,
  // B[k] = (Z[k] - conj Z[n-k]) / (2i) into the staged rows
  C *out = reinterpret_cast<C *>(stage) + 2 * ln.c * a.sp;
  const int second_out = 2 * units * a.sp;
  for (int k = ln.b0; k < a.nh; k += ln.step) {
    const int kr = k == 0 ? 0 : nk - k;
    const V p = ucmul<false>(tile[(k << a.lu) + ln.c], __ldg(a.chirp + k));
    const V q = ucmul<false>(tile[(kr << a.lu) + ln.c], __ldg(a.chirp + kr));
    const T h = (T)0.5;
    auto emit = [&](C *o, C zp, C zq) {
      o[k] = mk(h * (zp.x + zq.x), h * (zp.y - zq.y));
      o[k + a.sp] = mk(h * (zp.y + zq.y), h * (zq.x - zp.x));
    };
    if constexpr (CU == 1) {
      emit(out, p, q);
    } else {
      emit(out, p.a, q.a);
      emit(out + second_out, p.b, q.b);
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  rows_out(reinterpret_cast<unsigned char *>(spec + line0 * a.nhp), a.nhp * sizeof(C), stage, a.sp * sizeof(C), nl);
}

// C2R along z (ParisPencil.cpp:368-380).
template <typename T>
__global__ void __launch_bounds__(256, 3)
    k_bs_zinv(const typename Cplx<T>::type *spec, T *__restrict__ f,
              const __grid_constant__ BsPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / sizeof(C);
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t mbar;
  const int nk = a.nk, units = 1 << a.lu, lines = 2 * CU * units;
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
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  z_rows_real_ends(a, rows, nl, lines);
  __syncthreads();
  const GenLane ln = bs_lane(a);
  const C *ra = rows + 2 * ln.c * a.sp;
  const int second = 2 * units * a.sp;
  // the Hermitian extension times conj chirp, zero from nk on
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if (pos < nk) v[r] = ucmul<true>(z_extend<V>(ra, second, a.sp, nk, pos), __ldg(a.chirp + pos));
      else v[r] = zero_unit((V *)nullptr);
    }
  };
  // points k < n, times conj chirp, to the real lines of the pairs
  T *out = reinterpret_cast<T *>(stage) + 2 * ln.c * a.lp;
  const int second_out = 2 * units * a.lp;
  auto put = [&](int, int pos0, const GenStage &st, const V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = pos0 + r * st.m;
      if (k < nk) {
        const V z = ucmul<true>(v[r], __ldg(a.chirp + k));
        T *o = out + k;
        if constexpr (CU == 1) {
          o[0] = z.x;
          o[a.lp] = z.y;
        } else {
          o[0] = z.a.x;
          o[a.lp] = z.a.y;
          o[second_out] = z.b.x;
          o[second_out + a.lp] = z.b.y;
        }
      }
    }
  };
  bs_conv<BsWay, true>(a, ln, tile, ld0, put);
  fence_proxy_async_smem();
  __syncthreads();
  if (a.per_line)
    rows_out(reinterpret_cast<unsigned char *>(f + line0 * nk), nk * sizeof(T), stage, a.lp * sizeof(T), nl);
  else
    bulk_out(f + line0 * nk, reinterpret_cast<const T *>(stage), (size_t)nl * nk);
}

// KIND 1: y forward, 3: y inverse (ParisPencil.cpp:173-212, :322-334); 2: x
// forward, filter, x inverse (:221-297, :406-421).  One tile of spectrum
// columns per block: y tiles are plane i = o with rows j (row stride nhp), x
// tiles plane j = o with rows i (row stride nj*nhp).
template <typename T, int KIND>
__global__ void __launch_bounds__(256, 3)
    k_bs_strided(const typename Cplx<T>::type *src, typename Cplx<T>::type *dst,
                 const __grid_constant__ BsPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / sizeof(C);
  extern __shared__ unsigned char smraw[];
  V *tile = reinterpret_cast<V *>(align128(smraw));
  pdl_start();
  pdl_wait();
  const int n = a.n;
  const int W = CU << a.lu;
  const int ktiles = (a.nh + W - 1) / W;
  const int o = blockIdx.x / ktiles;
  const int kt = blockIdx.x - o * ktiles;
  const GenLane ln = bs_lane(a);
  const int col = kt * W + ln.c * CU;
  // FP32 rows are padded to an even count: a unit whose second column is past
  // nh reads the padding and does not store it
  const bool live = col < a.nh, whole = CU == 1 || col + 1 < a.nh;
  const long pitch = KIND == 2 ? (long)a.nj * a.nhp : (long)a.nhp;
  const long base = (KIND == 2 ? (long)o * a.nhp : (long)o * a.nj * a.nhp) + col;
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      v[r] = pos < n && live ? *reinterpret_cast<const V *>(src + base + pos * pitch) : zero_unit((V *)nullptr);
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if (pos < n) v[r] = ucmul<KIND == 3>(v[r], __ldg(a.chirp + pos));
    }
  };
  auto put = [&](int, int pos0, const GenStage &st, const V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = pos0 + r * st.m;
      if (k < n && live) {
        const V z = ucmul<KIND != 1>(v[r], __ldg(a.chirp + k));
        C *p = dst + base + k * pitch;
        if (whole) *reinterpret_cast<V *>(p) = z;
        else if constexpr (CU == 2) *p = z.a;
      }
    }
  };
  if constexpr (KIND != 2) {
    bs_conv<BsWay, KIND == 3>(a, ln, tile, ld0, put);
  } else {
    const double jd = double(min(o, a.nj - o)) * a.dd[1];
    const double ka = double(col) * a.dd[2], kb = double(col + 1) * a.dd[2];
    const GenFilter flt{a.ni, o, col, jd * jd, a.dd[0], -a.invN, ka * ka, kb * kb};
    // The last forward stage leaves X[k] = chirp[k] conv[k]; the inverse
    // transform's input is X[k] d(k) conj chirp[k] = conv[k] d(k), as
    // |chirp| = 1, so that is what it stores (zero from n on).
    auto putf = [&](int row, int pos0, const GenStage &st, const V *v, auto tag) {
      constexpr int R = decltype(tag)::value;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int k = pos0 + r * st.m;
        V z = zero_unit((V *)nullptr);
        if (k < n) {
          z = v[r];
          flt.apply(k, z);
        }
        tile[((row + r * st.m) << a.lu) + ln.c] = z;
      }
    };
    bs_conv<BsWay, false>(a, ln, tile, ld0, putf);
    bs_conv<BsWay, true>(a, ln, tile, TileLoad<V>{tile, a.lu, ln.c}, put);
  }
}

// chirp[j] = exp(-i*pi*j^2/n): the exponent reduced exactly (j^2 mod 2n)
// before FP64 sincospi.
template <typename C> __global__ void k_bs_chirp(int n, C *chirp) {
  using R = typename Real<C>::type;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const long long q = (long long)j * j % (2LL * n);
    double s, c;
    sincospi((double)q / (double)n, &s, &c);
    chirp[j] = mk((R)c, (R)(-s));
  }
}

// ghat[pos] = G[k] / M for the frequency k at DIF position pos = g R + r, which
// is k0[g] + r M/R; G[k] = sum_m g[m] exp(-2*pi*i*m*k/M) over the wrapped kernel
// g[m] = g[M-m] = exp(+i*pi*m^2/n) (m < n):
//   G[k] = 1 + 2 sum_{m=1}^{n-1} exp(i*pi*m^2/n) cos(2*pi*m*k/M),
// a direct FP64 sum (exponents reduced exactly), in blocks of 32 terms.
template <typename C> __global__ void k_bs_ghat(int n, int M, const int *k0, int last_radix, C *ghat) {
  using R = typename Real<C>::type;
  for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < M; pos += gridDim.x * blockDim.x) {
    const int g = pos / last_radix;
    const int k = k0[g] + (pos - g * last_radix) * (M / last_radix);
    double gx = 1.0, gy = 0.0;
    for (int m0 = 1; m0 < n; m0 += 32) {
      double px = 0.0, py = 0.0;
      for (int m = m0; m < min(n, m0 + 32); m++) {
        const long long q = (long long)m * m % (2LL * n);
        const long long r = (long long)m * k % M;
        double s, c;
        sincospi((double)q / (double)n, &s, &c);
        const double cs = cospi(2.0 * (double)r / (double)M);
        px += c * cs;
        py += s * cs;
      }
      gx += 2.0 * px;
      gy += 2.0 * py;
    }
    ghat[pos] = mk((R)(gx / M), (R)(gy / M));
  }
}

template <typename T> const void *bs_kernel(int kind) {
  switch (kind) {
    case 0: return (const void *)k_bs_zfwd<T>;
    case 1: return (const void *)k_bs_strided<T, 1>;
    case 2: return (const void *)k_bs_strided<T, 2>;
    case 3: return (const void *)k_bs_strided<T, 3>;
    default: return (const void *)k_bs_zinv<T>;
  }
}

}  // namespace

// The cheapest 2^a 3^b 5^c 7^d length from 2n - 1 to a third more, by the cost
// of its stages (a length of fewer, better radices is worth some padding: 251
// points go through 512 = 8 x 8 x 8, not 504 = 8 x 7 x 9); above 1500 points the
// smallest, whose tile has to fit.
int bs_padded_length(int n) {
  const int lo = std::max(1, 2 * n - 1), hi = n > 1500 ? lo : lo + lo / 3;
  int best = 0;
  double cost = 0.0;
  for (int m = lo; m <= hi || best == 0; m++) {
    if (!smooth2357(m)) continue;
    const double c = m * gen_cost(m);
    if (best == 0 || c < cost) {
      best = m;
      cost = c;
    }
  }
  return best;
}

GenShape bs_shape(int kind, int ni, int nj, int nk, int nhp, int esz, int M, int num_sms) {
  GenShape s{};
  const int cu = 16 / (2 * esz);
  if (kind == 0 || kind == 4) {
    s.tile_rows = M;
    gen_z_shape(&s, ni, nj, nk, nhp, esz, num_sms, false);
    return s;
  }
  const int nh = nk / 2 + 1;
  for (s.units = 8;; s.units /= 2) {
    s.smem = (size_t)M * s.units * 16 + 128;
    const int w = s.units * cu;
    s.grid = (long)(kind == 2 ? nj : ni) * ((nh + w - 1) / w);
    if (s.units == 2) break;
    if (s.units == 8 ? s.smem <= 74 * 1024 && s.grid >= num_sms : s.smem <= 112 * 1024) break;
  }
  gen_pick_threads(&s);
  return s;
}

template <typename T> int bs_prepare(int kind, size_t smem) {
  size_t avail = 0;
  const int rc = allow_dyn_smem_fn(bs_kernel<T>(kind), &avail);
  if (rc != FF_OK) return rc;
  if (smem > avail)
    return set_error(FF_ERR_UNSUPPORTED, "Bluestein tile of %zu bytes does not fit in shared memory", smem);
  return FF_OK;
}

template <typename C> int bs_tables(int n, int M, const int *k0, int last_radix, C *chirp, C *ghat) {
  k_bs_chirp<<<std::min(1024, (n + 255) / 256), 256>>>(n, chirp);
  k_bs_ghat<<<std::min(1024, (M + 127) / 128), 128>>>(n, M, k0, last_radix, ghat);
  FF_CUDA(cudaGetLastError());
  return FF_OK;
}

template <typename T>
int bs_launch(int kind, const BsPass<typename Cplx<T>::type> &a, const GenShape &s, const void *in, void *out,
              cudaStream_t st) {
  using C = typename Cplx<T>::type;
  const C *ci = static_cast<const C *>(in);
  C *co = static_cast<C *>(out);
  auto go = [&](auto k, auto... args) { return launch_chained(s.chained, k, (unsigned)s.grid, s.threads, s.smem, st, args...); };
  cudaError_t e;
  switch (kind) {
    case 0: e = go(k_bs_zfwd<T>, static_cast<const T *>(in), co, a); break;
    case 1: e = go(k_bs_strided<T, 1>, ci, co, a); break;
    case 2: e = go(k_bs_strided<T, 2>, ci, co, a); break;
    case 3: e = go(k_bs_strided<T, 3>, ci, co, a); break;
    default: e = go(k_bs_zinv<T>, ci, static_cast<T *>(out), a); break;
  }
  FF_CUDA(e);
  return FF_OK;
}

template int bs_prepare<double>(int, size_t);
template int bs_prepare<float>(int, size_t);
template int bs_tables<double2>(int, int, const int *, int, double2 *, double2 *);
template int bs_tables<float2>(int, int, const int *, int, float2 *, float2 *);
template int bs_launch<double>(int, const BsPass<double2> &, const GenShape &, const void *, void *, cudaStream_t);
template int bs_launch<float>(int, const BsPass<float2> &, const GenShape &, const void *, void *, cudaStream_t);

}  // namespace ff
