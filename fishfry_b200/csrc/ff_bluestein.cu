// Passes of the single-grid solve for axes with a prime factor above 7 by
// Rader's or Bluestein's algorithm (both and their tables are described in
// ff_bluestein.hpp).
//
// One kernel per pass kind and algorithm, on the stages of the generic passes
// (16-byte units, radices up to 10, plan read at run time):
//   z forward / inverse: `units` columns of line pairs per block; the lines
//     arrive in a staging area by bulk copies and the result leaves from it;
//   y forward / inverse, x: `units` spectrum columns x M rows per block, rows
//     read and written directly from HBM (not the box a TMA copy would move:
//     Bluestein's tile holds M > n rows, Rader's holds them permuted).
// The x kernel runs the forward transform, stores the filtered spectrum in
// place through its last stage, and runs the inverse on the same tile.
//
// Each direction is two M-point transforms: the passes are bound by their stages
// (instruction issue and shared memory), not by HBM, so they go by M.  Bluestein
// needs M >= 2n - 1 and takes the cheapest smooth length, not the smallest
// (bs_padded_length); Rader's M is n - 1, half of that, without the chirps, for the
// primes that allow it.  One B200, passes z / y / x / y / z, all through Bluestein
// and now: 211^3 FP64 121 / 120 / 209 / 115 / 127 us -> 85 / 76 / 121 / 75 / 82, FP32
// 73 / 66 / 119 / 64 / 78 -> 47 / 56 / 100 / 54 / 47; 256x256x251 z FP64 255 / 259
// -> 123 / 121, FP32 132 / 133 -> 71 / 74; 401^3 FP64 sum 5370 -> 2630.

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
// RADER: tile row N holds the line's point 0, written and read by the lane of
// butterfly 0; the sum of the others is the transform's frequency 0, so that lane
// adds it there (the result's point 0) and adds point 0 to every output through
// the product's frequency 0.
template <typename WAY, bool RADER, bool INV, typename V, typename C, typename LD0, typename ST>
__device__ __forceinline__ void bs_conv(const BsPass<C> &a, const GenLane &ln, V *tile, LD0 &&ld0, ST &&put) {
  const GenAxis<C> &ax = a.ax;
  const int S = ax.S;   // at least two stages (M >= 21; Rader from 13 points on)
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
      const V sum = v[0];
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = ucmul<INV>(v[r], __ldg(a.ghat + b * R + r));
      if (RADER && b == 0) {
        V &first = tile[(ax.n << a.lu) + ln.c];
        v[0] = uadd(v[0], first);
        first = uadd(first, sum);
      }
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

// The line's index of the convolution's input q (IN) or output q: the line itself
// (Bluestein), or its points but 0 in the order of powers of the root g of BsPass
// (Rader): the forward transform reads g^q and gives g^-q, the inverse reads g^-q
// and gives g^q.
template <bool RADER, bool POWER, typename C> __device__ __forceinline__ int bs_at(const BsPass<C> &a, int q) {
  if constexpr (!RADER) return q;
  else return __ldg(a.perm + (POWER || q == 0 ? q : a.ax.n - q));
}

// R2C along z (ParisPencil.cpp:152-165).
template <typename T, bool RADER>
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
  const GenLane ln = gen_lane(a);
  const T *ra = raw + 2 * ln.c * a.lp;
  const int second = 2 * units * a.lp;
  // point `pos` of two real lines as one complex line
  auto pair = [&](int pos) { return unit_of<V>(ra + pos, a.lp, second); };
  // Rader: in the root's order; Bluestein: times the chirp, zero from nk on
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if constexpr (RADER) v[r] = pair(bs_at<true, true>(a, pos));
      else if (pos < nk) v[r] = ucmul<false>(pair(pos), __ldg(a.chirp + pos));
      else v[r] = zero_unit((V *)nullptr);
    }
  };
  if (RADER && ln.b0 == 0) tile[(a.ax.n << a.lu) + ln.c] = pair(0);
  bs_conv<BsWay, RADER, false>(a, ln, tile, ld0, TilePut<V>{tile, a.lu, ln.c});
  // Z[k] = chirp[k] conv[k]; A[k] = (Z[k] + conj Z[n-k]) / 2,
  // B[k] = (Z[k] - conj Z[n-k]) / (2i) into the staged rows.  Rader: row q holds
  // Z[k], k = g^-q, and row q + N/2 its Z[n-k], as g^(N/2) = -1.
  C *out = reinterpret_cast<C *>(stage) + 2 * ln.c * a.sp;
  const int second_out = 2 * units * a.sp;
  for (int i = ln.b0; i < a.nh; i += ln.step) {
    int k = i;
    V p, q;
    if constexpr (RADER) {
      const int N = a.ax.n;
      const V s = tile[((i == 0 ? N : i - 1) << a.lu) + ln.c];
      const V t = tile[((i == 0 ? N : i - 1 + N / 2) << a.lu) + ln.c];
      k = i == 0 ? 0 : bs_at<true, false>(a, i - 1);
      const bool low = 2 * k <= nk;
      if (!low) k = nk - k;
      p = low ? s : t;
      q = low ? t : s;
    } else {
      const int kr = k == 0 ? 0 : nk - k;
      p = ucmul<false>(tile[(k << a.lu) + ln.c], __ldg(a.chirp + k));
      q = ucmul<false>(tile[(kr << a.lu) + ln.c], __ldg(a.chirp + kr));
    }
    unit_split(out + k, a.sp, second_out, p, q);
  }
  fence_proxy_async_smem();
  __syncthreads();
  rows_out(reinterpret_cast<unsigned char *>(spec + line0 * a.nhp), a.nhp * sizeof(C), stage, a.sp * sizeof(C), nl);
}

// C2R along z (ParisPencil.cpp:368-380).
template <typename T, bool RADER>
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
  const GenLane ln = gen_lane(a);
  const C *ra = rows + 2 * ln.c * a.sp;
  const int second = 2 * units * a.sp;
  // the Hermitian extension (Bluestein: times conj chirp, zero from nk on)
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if constexpr (RADER) v[r] = unit_extend<V>(ra, a.sp, second, nk, bs_at<true, false>(a, pos));
      else if (pos < nk) v[r] = ucmul<true>(unit_extend<V>(ra, a.sp, second, nk, pos), __ldg(a.chirp + pos));
      else v[r] = zero_unit((V *)nullptr);
    }
  };
  // points k < n (Bluestein: times conj chirp) to the real lines of the pairs
  T *out = reinterpret_cast<T *>(stage) + 2 * ln.c * a.lp;
  const int second_out = 2 * units * a.lp;
  auto store = [&](int k, V z) { unit_put(out + k, a.lp, second_out, z); };
  auto put = [&](int, int pos0, const GenStage &st, const V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = pos0 + r * st.m;
      if constexpr (RADER) store(bs_at<true, true>(a, k), v[r]);
      else if (k < nk) store(k, ucmul<true>(v[r], __ldg(a.chirp + k)));
    }
  };
  V *first = tile + (a.ax.n << a.lu) + ln.c;
  if (RADER && ln.b0 == 0) *first = unit_extend<V>(ra, a.sp, second, nk, 0);
  bs_conv<BsWay, RADER, true>(a, ln, tile, ld0, put);
  if (RADER && ln.b0 == 0) store(0, *first);
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
template <typename T, int KIND, bool RADER>
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
  const GenLane ln = gen_lane(a);
  const int col = kt * W + ln.c * CU;
  // FP32 rows are padded to an even count: a unit whose second column is past
  // nh reads the padding and does not store it
  const bool live = col < a.nh, whole = CU == 1 || col + 1 < a.nh;
  const long pitch = KIND == 2 ? (long)a.nj * a.nhp : (long)a.nhp;
  const long base = (KIND == 2 ? (long)o * a.nhp : (long)o * a.nj * a.nhp) + col;
  auto row_in = [&](int pos) -> V {
    return live ? *reinterpret_cast<const V *>(src + base + pos * pitch) : zero_unit((V *)nullptr);
  };
  auto row_out = [&](int k, V z) {
    C *p = dst + base + k * pitch;
    if (whole) *reinterpret_cast<V *>(p) = z;
    else if constexpr (CU == 2) *p = z.a;
  };
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      if constexpr (RADER) v[r] = row_in(bs_at<true, KIND != 3>(a, pos));
      else v[r] = pos < n ? row_in(pos) : zero_unit((V *)nullptr);
    }
    if constexpr (!RADER) {
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int pos = pos0 + r * st.m;
        if (pos < n) v[r] = ucmul<KIND == 3>(v[r], __ldg(a.chirp + pos));
      }
    }
  };
  auto put = [&](int, int pos0, const GenStage &st, const V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int k = pos0 + r * st.m;
      if constexpr (RADER) {
        if (live) row_out(bs_at<true, KIND != 1>(a, k), v[r]);
      } else if (k < n && live) {
        row_out(k, ucmul<KIND != 1>(v[r], __ldg(a.chirp + k)));
      }
    }
  };
  V *first = tile + (a.ax.n << a.lu) + ln.c;
  if (RADER && ln.b0 == 0) *first = row_in(0);
  if constexpr (KIND != 2) {
    bs_conv<BsWay, RADER, KIND == 3>(a, ln, tile, ld0, put);
  } else {
    const double jd = double(min(o, a.nj - o)) * a.dd[1];
    const double ka = double(col) * a.dd[2], kb = double(col + 1) * a.dd[2];
    const GenFilter flt{a.ni, o, col, jd * jd, a.dd[0], -a.invN, ka * ka, kb * kb};
    // Bluestein: the last forward stage leaves X[k] = chirp[k] conv[k]; the inverse
    // transform's input is X[k] d(k) conj chirp[k] = conv[k] d(k), as
    // |chirp| = 1, so that is what it stores (zero from n on).  Rader: the
    // forward transform's order is the inverse one's input order.
    auto putf = [&](int row, int pos0, const GenStage &st, const V *v, auto tag) {
      constexpr int R = decltype(tag)::value;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int k = pos0 + r * st.m;
        V z = zero_unit((V *)nullptr);
        if (RADER || k < n) {
          z = v[r];
          flt.apply(bs_at<RADER, false>(a, k), z);
        }
        tile[((row + r * st.m) << a.lu) + ln.c] = z;
      }
    };
    bs_conv<BsWay, RADER, false>(a, ln, tile, ld0, putf);
    if (RADER && ln.b0 == 0) {
      V z = *first;
      flt.apply(0, z);
      *first = z;
    }
    bs_conv<BsWay, RADER, true>(a, ln, tile, TileLoad<V>{tile, a.lu, ln.c}, put);
  }
  if (RADER && ln.b0 == 0 && live) row_out(0, *first);
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

// ghat of Rader's convolution of N = n - 1 points: at DIF position pos, G[k] / N
// for its frequency k, G[k] = sum_m exp(-2*pi*i*g^-m/n) exp(-2*pi*i*m*k/N), a direct
// FP64 sum (exponents reduced exactly) in blocks of 32 terms.  perm[q] = g^q mod n.
template <typename C>
__global__ void k_rader_ghat(int n, const int *perm, const int *k0, int last_radix, C *ghat) {
  using R = typename Real<C>::type;
  const int N = n - 1;
  for (int pos = blockIdx.x * blockDim.x + threadIdx.x; pos < N; pos += gridDim.x * blockDim.x) {
    const int g = pos / last_radix;
    const int k = k0[g] + (pos - g * last_radix) * (N / last_radix);
    double gx = 0.0, gy = 0.0;
    for (int m0 = 0; m0 < N; m0 += 32) {
      double px = 0.0, py = 0.0;
      for (int m = m0; m < min(N, m0 + 32); m++) {
        // the two factors' phases as one fraction of n N
        const long long q = (long long)perm[m == 0 ? 0 : N - m] * N + (long long)m * k % N * n;
        double s, c;
        sincospi(2.0 * (double)(q % ((long long)n * N)) / ((double)n * (double)N), &s, &c);
        px += c;
        py -= s;
      }
      gx += px;
      gy += py;
    }
    ghat[pos] = mk((R)(gx / N), (R)(gy / N));
  }
}

template <typename T, bool RADER> const void *bs_kernel(int kind) {
  switch (kind) {
    case 0: return (const void *)k_bs_zfwd<T, RADER>;
    case 1: return (const void *)k_bs_strided<T, 1, RADER>;
    case 2: return (const void *)k_bs_strided<T, 2, RADER>;
    case 3: return (const void *)k_bs_strided<T, 3, RADER>;
    default: return (const void *)k_bs_zinv<T, RADER>;
  }
}

}  // namespace

int rader_root(int n) {
  if (n < 13 || !smooth2357(n - 1)) return 0;
  for (int q = 2; q * q <= n; q++)
    if (n % q == 0) return 0;
  // the smallest g whose powers g^((n-1)/p) are not 1 for the primes p of n - 1
  for (int g = 2;; g++) {
    bool root = true;
    for (int p : {2, 3, 5, 7}) {
      if ((n - 1) % p != 0) continue;
      long long v = 1;
      for (int e = 0; e < (n - 1) / p; e++) v = v * g % n;
      root = root && v != 1;
    }
    if (root) return g;
  }
}

// The cheapest 2^a 3^b 5^c 7^d length from 2n - 1 to a third more, by the cost
// of its stages (a length of fewer, better radices is worth some padding: from 501
// on 512 = 8 x 8 x 8, not 504 = 9 x 8 x 7); above 1500 points the
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

GenShape bs_shape(int kind, int ni, int nj, int nk, int nhp, int esz, int rows, int num_sms) {
  GenShape s{};
  const int cu = 16 / (2 * esz);
  if (kind == 0 || kind == 4) {
    s.tile_rows = rows;
    // larger tiles than the generic z passes take: these are bound by their stages,
    // and rows of few units (two at M = 512) put the last stage's butterflies in
    // the same banks.  z passes at 40 KB -> here, FP64: 254^3 251 / 257 -> 217 /
    // 221 us, 256x256x251 133 / 125 -> 123 / 121, 211^3 85 / 77 -> 85 / 82; FP32:
    // 254^3 129 / 131 -> 118 / 119, 401^3 257 / 253 -> 254 / 243, 211^3 45 -> 47
    gen_z_shape(&s, ni, nj, nk, nhp, esz, num_sms, false, (esz == 8 ? 76 : 56) * 1024);
    return s;
  }
  const int nh = nk / 2 + 1;
  for (s.units = 8;; s.units /= 2) {
    s.smem = (size_t)rows * s.units * 16 + 128;
    const int w = s.units * cu;
    s.grid = (long)(kind == 2 ? nj : ni) * ((nh + w - 1) / w);
    if (s.units == 2) break;
    if (s.units == 8 ? s.smem <= 74 * 1024 && s.grid >= num_sms : s.smem <= 112 * 1024) break;
  }
  gen_pick_threads(&s);
  return s;
}

template <typename T> int bs_prepare(int kind, bool rader, size_t smem) {
  size_t avail = 0;
  const int rc = allow_dyn_smem_fn(rader ? bs_kernel<T, true>(kind) : bs_kernel<T, false>(kind), &avail);
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

template <typename C> int rader_tables(int n, const int *perm, const int *k0, int last_radix, C *ghat) {
  k_rader_ghat<<<std::min(1024, (n + 127) / 128), 128>>>(n, perm, k0, last_radix, ghat);
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
  auto launch = [&](auto rader) {
    constexpr bool RADER = decltype(rader)::value;
    switch (kind) {
      case 0: return go(k_bs_zfwd<T, RADER>, static_cast<const T *>(in), co, a);
      case 1: return go(k_bs_strided<T, 1, RADER>, ci, co, a);
      case 2: return go(k_bs_strided<T, 2, RADER>, ci, co, a);
      case 3: return go(k_bs_strided<T, 3, RADER>, ci, co, a);
      default: return go(k_bs_zinv<T, RADER>, ci, static_cast<T *>(out), a);
    }
  };
  FF_CUDA(a.perm ? launch(std::true_type{}) : launch(std::false_type{}));
  return FF_OK;
}

template int bs_prepare<double>(int, bool, size_t);
template int bs_prepare<float>(int, bool, size_t);
template int rader_tables<double2>(int, const int *, const int *, int, double2 *);
template int rader_tables<float2>(int, const int *, const int *, int, float2 *);
template int bs_tables<double2>(int, int, const int *, int, double2 *, double2 *);
template int bs_tables<float2>(int, int, const int *, int, float2 *, float2 *);
template int bs_launch<double>(int, const BsPass<double2> &, const GenShape &, const void *, void *, cudaStream_t);
template int bs_launch<float>(int, const BsPass<float2> &, const GenShape &, const void *, void *, cudaStream_t);

}  // namespace ff
