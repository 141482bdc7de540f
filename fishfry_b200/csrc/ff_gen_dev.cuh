// Kernels of the passes along axes without a compile-time plan.  Included by
// ff_gen_f64.cu and ff_gen_f32.cu, one precision each.
//
// Every tile is point-major in units of 16 bytes: [row][unit], a unit being one
// FP64 or two adjacent FP32 complex columns (z passes: one FP64 line pair or
// two FP32 ones, as complex lines), so both precisions run the same code on
// 16-byte shared-memory accesses.  Threads take units fastest: a thread keeps
// its unit, and walks butterflies b0, b0 + step, ... of that column.
//
// What bounded these passes before was integer work of the plan read at run
// time: 338 (z) and 180 (y) warp instructions per 32 complex points at
// 480x400x360 FP64, a fifth of them FP64 (a digit reversal with a remainder by
// the runtime radix for each output, a quotient for each butterfly, five-factor
// plans).  So here
//   - radices go up to 10 (6 and 10 without inner twiddles, by the prime factor
//     algorithm), which makes three stages of nearly every length up to 1000;
//   - the butterfly's block and offset advance by additions;
//   - a butterfly's points are one pointer and a uniform stride on both sides
//     (the last stage of a forward transform has frequencies k0 + r n/R, so its
//     stores to HBM or to staged rows are one too): one table load per group;
//   - twiddles lie per stage as [j][r], one address for a butterfly's factors;
//   - the z passes fuse the last stage with the real split as the compile-time
//     ones do, in one form for every radix.
// One B200, passes z / y / x / y / z: 480x400x360 FP64 483 / 328 / 424 / 326 /
// 581 us before, 243 / 215 / 324 / 211 / 240 now (2.14 -> 1.23 ms a solve, 70 %
// of the copy rate over the five passes' bytes); FP32 332 / 229 / 301 / 232 / 369
// -> 162 / 137 / 206 / 138 / 160 us (1.46 -> 0.80 ms).
//
// What bounds them now: no pipe is saturated (480x400x360 FP64 y pass: DRAM 60 %,
// L1 55 %, FP64 32 %, issue 37 %); a block's load, its stages and its stores
// follow one another, and 24 warps on an SM (80 registers) overlap them across
// blocks.  Persistent blocks with two tile buffers, so that no warp waits for a
// load, need blocks of twice the size, half as many: their warps then load, add
// and store in step, which cost more than it hid (y 217 -> 290, x 335 -> 417,
// z 245 -> 350 us).  64 registers and 32 warps spill (y 217 -> 247 us).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "ff_gen.hpp"
#include "ff_status.hpp"
#include "ff_tiles.cuh"

namespace ff {

// Two adjacent FP32 complex columns.
struct __align__(16) FPair {
  float2 a, b;
};
template <typename C> struct Unit;
template <> struct Unit<double2> { using type = double2; };
template <> struct Unit<float2> { using type = FPair; };

// ---------------------------------------------------------------- arithmetic
__device__ __forceinline__ double2 uadd(double2 a, double2 b) { return mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 usub(double2 a, double2 b) { return mk(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 uscale(double2 a, double s) { return mk(a.x * s, a.y * s); }
// c + s*a
__device__ __forceinline__ double2 ufma(double2 a, double s, double2 c) {
  return mk(fma(a.x, s, c.x), fma(a.y, s, c.y));
}
template <bool INV> __device__ __forceinline__ double2 umul_wi(double2 a) { return mul_wi<INV>(a); }
template <bool CONJ> __device__ __forceinline__ double2 ucmul(double2 a, double2 w) {
  return CONJ ? cmulc(a, w) : cmul(a, w);
}

__device__ __forceinline__ FPair uadd(FPair a, FPair b) { return {__fadd2_rn(a.a, b.a), __fadd2_rn(a.b, b.b)}; }
__device__ __forceinline__ FPair usub(FPair a, FPair b) {
  const float2 m = make_float2(-1.0f, -1.0f);
  return {__ffma2_rn(b.a, m, a.a), __ffma2_rn(b.b, m, a.b)};
}
__device__ __forceinline__ FPair uscale(FPair a, float s) {
  const float2 v = make_float2(s, s);
  return {__fmul2_rn(a.a, v), __fmul2_rn(a.b, v)};
}
__device__ __forceinline__ FPair ufma(FPair a, float s, FPair c) {
  const float2 v = make_float2(s, s);
  return {__ffma2_rn(a.a, v, c.a), __ffma2_rn(a.b, v, c.b)};
}
template <bool INV> __device__ __forceinline__ FPair umul_wi(FPair a) { return {mul_wi<INV>(a.a), mul_wi<INV>(a.b)}; }
template <bool CONJ> __device__ __forceinline__ FPair ucmul(FPair a, float2 w) {
  return CONJ ? FPair{cmulc(a.a, w), cmulc(a.b, w)} : FPair{cmul(a.a, w), cmul(a.b, w)};
}

template <typename V> struct UReal;
template <> struct UReal<double2> { using type = double; };
template <> struct UReal<FPair> { using type = float; };

// cos and sin of 2 pi k / 9, k = 1, 2, 4, to 40 digits
#define FF_C9_1 0.76604444311897803520239265055541667394
#define FF_S9_1 0.64278760968653932632264340990726343291
#define FF_C9_2 0.17364817766693034885171662676931479600
#define FF_S9_2 0.98480775301220805936674302458952301367
#define FF_C9_4 (-0.93969262078590838405410927732473146994)
#define FF_S9_4 0.34202014332566873304409961468225958076

// In-register R-point DFT of units, y_s = sum_r v_r exp(-+2 pi i r s / R).
template <int R, bool INV, typename V> struct UDft;
template <bool INV, typename V> struct UDft<1, INV, V> {
  static __device__ __forceinline__ void run(V *) {}
};
template <bool INV, typename V> struct UDft<2, INV, V> {
  static __device__ __forceinline__ void run(V *v) {
    const V a = v[0], b = v[1];
    v[0] = uadd(a, b);
    v[1] = usub(a, b);
  }
};
template <bool INV, typename V> __device__ __forceinline__ void udft3(V &v0, V &v1, V &v2) {
  using T = typename UReal<V>::type;
  const V t = uadd(v1, v2);
  const V u = umul_wi<INV>(uscale(usub(v1, v2), (T)FF_SQRT3_2));
  const V m = ufma(t, (T)-0.5, v0);
  v0 = uadd(v0, t);
  v1 = uadd(m, u);
  v2 = usub(m, u);
}
template <bool INV, typename V> __device__ __forceinline__ void udft4(V &v0, V &v1, V &v2, V &v3) {
  const V t0 = uadd(v0, v2), t1 = usub(v0, v2);
  const V t2 = uadd(v1, v3), t3 = umul_wi<INV>(usub(v1, v3));
  v0 = uadd(t0, t2);
  v2 = usub(t0, t2);
  v1 = uadd(t1, t3);
  v3 = usub(t1, t3);
}
template <bool INV, typename V> __device__ __forceinline__ void udft5(V &v0, V &v1, V &v2, V &v3, V &v4) {
  using T = typename UReal<V>::type;
  const V t1 = uadd(v1, v4), t2 = uadd(v2, v3);
  const V t3 = usub(v1, v4), t4 = usub(v2, v3);
  const V b1 = ufma(t2, (T)FF_C5_2, ufma(t1, (T)FF_C5_1, v0));
  const V b2 = ufma(t2, (T)FF_C5_1, ufma(t1, (T)FF_C5_2, v0));
  const V d1 = umul_wi<INV>(ufma(t4, (T)FF_S5_2, uscale(t3, (T)FF_S5_1)));
  const V d2 = umul_wi<INV>(ufma(t4, (T)-FF_S5_1, uscale(t3, (T)FF_S5_2)));
  v0 = uadd(v0, uadd(t1, t2));
  v1 = uadd(b1, d1);
  v4 = usub(b1, d1);
  v2 = uadd(b2, d2);
  v3 = usub(b2, d2);
}
template <bool INV, typename V> struct UDft<3, INV, V> {
  static __device__ __forceinline__ void run(V *v) { udft3<INV>(v[0], v[1], v[2]); }
};
template <bool INV, typename V> struct UDft<4, INV, V> {
  static __device__ __forceinline__ void run(V *v) { udft4<INV>(v[0], v[1], v[2], v[3]); }
};
template <bool INV, typename V> struct UDft<5, INV, V> {
  static __device__ __forceinline__ void run(V *v) { udft5<INV>(v[0], v[1], v[2], v[3], v[4]); }
};
// 6 = 2 x 3 and 10 = 2 x 5 by the prime factor algorithm (Good 1958): input
// r = (N2 r1 + N1 r2) mod N, output s with s = s1 mod N1 and s = s2 mod N2, no
// factors between the two transforms.
template <bool INV, typename V> struct UDft<6, INV, V> {
  static __device__ __forceinline__ void run(V *v) {
    V e[3], o[3];   // s1 = 0, 1
#pragma unroll
    for (int q = 0; q < 3; q++) {
      e[q] = uadd(v[(2 * q) % 6], v[(3 + 2 * q) % 6]);
      o[q] = usub(v[(2 * q) % 6], v[(3 + 2 * q) % 6]);
    }
    udft3<INV>(e[0], e[1], e[2]);
    udft3<INV>(o[0], o[1], o[2]);
#pragma unroll
    for (int s = 0; s < 6; s++) v[s] = s % 2 ? o[s % 3] : e[s % 3];
  }
};
template <bool INV, typename V> struct UDft<10, INV, V> {
  static __device__ __forceinline__ void run(V *v) {
    V e[5], o[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      e[q] = uadd(v[(2 * q) % 10], v[(5 + 2 * q) % 10]);
      o[q] = usub(v[(2 * q) % 10], v[(5 + 2 * q) % 10]);
    }
    udft5<INV>(e[0], e[1], e[2], e[3], e[4]);
    udft5<INV>(o[0], o[1], o[2], o[3], o[4]);
#pragma unroll
    for (int s = 0; s < 10; s++) v[s] = s % 2 ? o[s % 5] : e[s % 5];
  }
};
template <bool INV, typename V> struct UDft<7, INV, V> {
  static __device__ __forceinline__ void run(V *v) {
    using T = typename UReal<V>::type;
    const V t1 = uadd(v[1], v[6]), t2 = uadd(v[2], v[5]), t3 = uadd(v[3], v[4]);
    const V u1 = usub(v[1], v[6]), u2 = usub(v[2], v[5]), u3 = usub(v[3], v[4]);
    const T c1 = (T)FF_C7_1, c2 = (T)FF_C7_2, c3 = (T)FF_C7_3;
    const T s1 = (T)FF_S7_1, s2 = (T)FF_S7_2, s3 = (T)FF_S7_3;
    const V b1 = ufma(t3, c3, ufma(t2, c2, ufma(t1, c1, v[0])));
    const V b2 = ufma(t3, c1, ufma(t2, c3, ufma(t1, c2, v[0])));
    const V b3 = ufma(t3, c2, ufma(t2, c1, ufma(t1, c3, v[0])));
    const V d1 = umul_wi<INV>(ufma(u3, s3, ufma(u2, s2, uscale(u1, s1))));
    const V d2 = umul_wi<INV>(ufma(u3, -s1, ufma(u2, -s3, uscale(u1, s2))));
    const V d3 = umul_wi<INV>(ufma(u3, s2, ufma(u2, -s1, uscale(u1, s3))));
    v[0] = uadd(v[0], uadd(t1, uadd(t2, t3)));
    v[1] = uadd(b1, d1);
    v[6] = usub(b1, d1);
    v[2] = uadd(b2, d2);
    v[5] = usub(b2, d2);
    v[3] = uadd(b3, d3);
    v[4] = usub(b3, d3);
  }
};
template <bool INV, typename V> struct UDft<8, INV, V> {
  static __device__ __forceinline__ void run(V *v) {
    using T = typename UReal<V>::type;
    udft4<INV>(v[0], v[2], v[4], v[6]);   // even points: y0, y1, y2, y3 in v[0], v[2], v[4], v[6]
    udft4<INV>(v[1], v[3], v[5], v[7]);
    // w8^s = exp(-+i pi s / 4): (o -+ i o)/sqrt 2, -+i, ...
    const T h = (T)FF_SQRT1_2;
    const V o1 = uscale(uadd(v[3], umul_wi<INV>(v[3])), h);
    const V o2 = umul_wi<INV>(v[5]);
    const V o3 = uscale(usub(umul_wi<INV>(v[7]), v[7]), h);
    const V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = uadd(e0, o0);
    v[4] = usub(e0, o0);
    v[1] = uadd(e1, o1);
    v[5] = usub(e1, o1);
    v[2] = uadd(e2, o2);
    v[6] = usub(e2, o2);
    v[3] = uadd(e3, o3);
    v[7] = usub(e3, o3);
  }
};
// 9 = 3 x 3: r = r1 + 3 r2, s = 3 s1 + s2, factors w9^(r1 s2) between.
template <bool INV, typename V> struct UDft<9, INV, V> {
  static __device__ __forceinline__ V rot(V v, double c, double s) {
    // v * (c -+ i s)
    using T = typename UReal<V>::type;
    return ufma(umul_wi<INV>(v), (T)s, uscale(v, (T)c));
  }
  static __device__ __forceinline__ void run(V *v) {
#pragma unroll
    for (int r = 0; r < 3; r++) udft3<INV>(v[r], v[r + 3], v[r + 6]);   // v[r + 3 s2]
    v[4] = rot(v[4], FF_C9_1, FF_S9_1);
    v[5] = rot(v[5], FF_C9_2, FF_S9_2);
    v[7] = rot(v[7], FF_C9_2, FF_S9_2);
    v[8] = rot(v[8], FF_C9_4, FF_S9_4);
#pragma unroll
    for (int s = 0; s < 3; s++) udft3<INV>(v[3 * s], v[3 * s + 1], v[3 * s + 2]);   // y[3 s1 + s2] in v[3 s2 + s1]
    const V y1 = v[3], y2 = v[6], y5 = v[7];
    v[3] = v[1];
    v[6] = v[2];
    v[7] = v[5];
    v[1] = y1;
    v[2] = y2;
    v[5] = y5;
  }
};

// --------------------------------------------------------------- one stage
// v[r] *= w^r (or conj) for the butterfly at offset j, from the stage's table:
// FP64 loads w (radices from 6 also w^h, h = R/2 rounded up, which halves the
// chain of products and its rounding) and forms the other powers (loading every
// factor measured slower), FP32 loads them two at a time.
template <int R, bool CONJ>
__device__ __forceinline__ void gen_twiddle(double2 *v, const double2 *__restrict__ t) {
  const double2 w1 = __ldg(t + 1);
  double2 w = w1;
  if constexpr (R < 6) {
#pragma unroll
    for (int r = 1; r < R; r++) {
      v[r] = ucmul<CONJ>(v[r], w);
      if (r + 1 < R) w = cmul(w, w1);
    }
  } else {
    constexpr int H = (R + 1) / 2;
    const double2 wh = __ldg(t + H);
    v[H] = ucmul<CONJ>(v[H], wh);
#pragma unroll
    for (int r = 1; r < H; r++) {
      v[r] = ucmul<CONJ>(v[r], w);
      if (H + r < R) v[H + r] = ucmul<CONJ>(v[H + r], cmul(wh, w));
      if (r + 1 < H) w = cmul(w, w1);
    }
  }
}
template <int R, bool CONJ> __device__ __forceinline__ void gen_twiddle(FPair *v, const float2 *__restrict__ t) {
  const float4 *t4 = reinterpret_cast<const float4 *>(t);
#pragma unroll
  for (int r = 0; r < R; r += 2) {
    const float4 w = __ldg(t4 + r / 2);
    if (r > 0) v[r] = ucmul<CONJ>(v[r], make_float2(w.x, w.y));
    if (r + 1 < R) v[r + 1] = ucmul<CONJ>(v[r + 1], make_float2(w.z, w.w));
  }
}

// The thread's place in a tile.
struct GenLane {
  int c;      // unit
  int b0;     // first butterfly
  int step;   // butterflies per round
};

// How a pass walks its tile: PAD, rows are padded (z passes, GenStage::ms); a
// thread takes butterflies of radix up to PAIR two at a time (FP64 strided
// passes: 480x400x360 x pass 335 -> 320 us; the z and FP32 passes lost 3-5 %).
template <bool PAD, int PAIR> struct GenWay {
  static constexpr bool kPad = PAD;
  static constexpr int kPair = PAIR;
};

// A stage in the tile (rows of 1 << lu units): ld(row, pos, v) fills the
// butterfly's R points (positions pos + r m, rows row + r ms), which go back to
// the same rows.  The thread walks its butterflies b0, b0 + step, ... of the
// column.
template <typename WAY, int R, bool INV, bool DIT, typename V, typename C, typename LD>
__device__ __forceinline__ void gen_stage(const GenStage &s, const C *__restrict__ tw, const GenLane &ln, V *tile,
                                          int lu, LD &&ld) {
  constexpr int RP = (R + 1) & ~1;
  const int stride = (WAY::kPad ? s.ms : s.m) << lu;
  int q = __float2int_rz((float)ln.b0 * s.inv_m);
  int j = ln.b0 - q * s.m;
  if (j < 0) { q--; j += s.m; }
  else if (j >= s.m) { q++; j -= s.m; }
  auto advance = [&] {
    q += s.dq;
    j += s.dr;
    if (j >= s.m) { j -= s.m; q++; }
  };
  // rows of the blocks of stage 0 are padded apart: one row each
  auto row_of = [&](int pos) { return WAY::kPad ? pos + __float2int_rz(((float)q + 0.5f) * s.inv_pb) : pos; };
  auto work = [&](V *v, int jj) {
    const C *t = tw + s.tw + jj * RP;
    if (DIT && s.m > 1) gen_twiddle<R, INV>(v, t);
    UDft<R, INV, V>::run(v);
    if (!DIT && s.m > 1) gen_twiddle<R, INV>(v, t);
  };
  auto put = [&](const V *v, int row) {
    V *p = tile + (row << lu) + ln.c;
#pragma unroll
    for (int r = 0; r < R; r++) p[r * stride] = v[r];
  };
  int b = ln.b0;
  if constexpr (R <= WAY::kPair) {
    for (; b + ln.step < s.nb; b += 2 * ln.step) {
      const int j1 = j, pos1 = q * s.L + j, row1 = row_of(pos1);
      advance();
      const int pos2 = q * s.L + j, row2 = row_of(pos2);
      V v[R], w[R];
      ld(row1, pos1, s, v, RadixTag<R>{});
      ld(row2, pos2, s, w, RadixTag<R>{});
      work(v, j1);
      work(w, j);
      put(v, row1);
      put(w, row2);
      advance();
    }
  }
  for (; b < s.nb; b += ln.step) {
    const int pos = q * s.L + j, row = row_of(pos);
    V v[R];
    ld(row, pos, s, v, RadixTag<R>{});
    work(v, j);
    put(v, row);
    advance();
  }
}

template <typename F> __device__ __forceinline__ void with_gen_radix(int r, F &&f) {
  switch (r) {
    case 2: f(RadixTag<2>{}); break;
    case 3: f(RadixTag<3>{}); break;
    case 4: f(RadixTag<4>{}); break;
    case 5: f(RadixTag<5>{}); break;
    case 6: f(RadixTag<6>{}); break;
    case 7: f(RadixTag<7>{}); break;
    case 8: f(RadixTag<8>{}); break;
    case 9: f(RadixTag<9>{}); break;
    case 10: f(RadixTag<10>{}); break;
    default: f(RadixTag<1>{}); break;
  }
}
// The last radix of the z passes (two groups per thread).
template <typename F> __device__ __forceinline__ void with_split_radix(int r, F &&f) {
  switch (r) {
    case 2: f(RadixTag<2>{}); break;
    case 3: f(RadixTag<3>{}); break;
    case 4: f(RadixTag<4>{}); break;
    case 5: f(RadixTag<5>{}); break;
    case 6: f(RadixTag<6>{}); break;
    case 7: f(RadixTag<7>{}); break;
    default: f(RadixTag<1>{}); break;
  }
}

// Loads from the tile itself: rows row + r stride.
template <typename V> struct TileLoad {
  const V *tile;
  int lu, c;
  template <int R> __device__ __forceinline__ void at(int row, int stride, V *v, RadixTag<R>) const {
    const V *p = tile + (row << lu) + c;
    const int step = stride << lu;
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = p[r * step];
  }
  template <int R>
  __device__ __forceinline__ void operator()(int row, int, const GenStage &s, V *v, RadixTag<R> tag) const {
    at(row, s.ms, v, tag);
  }
};

// DIF stages 0 .. s1-1 in the tile, each followed by a barrier; the first reads
// through ld0.
template <typename WAY, bool INV, typename V, typename C, typename LD0>
__device__ __forceinline__ void gen_dif(const GenAxis<C> &ax, int s1, const GenLane &ln, V *tile, int lu, LD0 &&ld0) {
  const TileLoad<V> ld{tile, lu, ln.c};
  for (int s = 0; s < s1; s++) {
    with_gen_radix(ax.st[s].R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      if constexpr (std::is_same<std::decay_t<LD0>, TileLoad<V>>::value) {
        gen_stage<WAY, R, INV, false>(ax.st[s], ax.tw, ln, tile, lu, ld);
      } else {
        if (s == 0) gen_stage<WAY, R, INV, false>(ax.st[s], ax.tw, ln, tile, lu, ld0);
        else gen_stage<WAY, R, INV, false>(ax.st[s], ax.tw, ln, tile, lu, ld);
      }
    });
    __syncthreads();
  }
}

template <typename C> __device__ __forceinline__ GenLane gen_lane(const GenPass<C> &a) {
  return {(int)threadIdx.x & ((1 << a.lu) - 1), (int)threadIdx.x >> a.lu, (int)blockDim.x >> a.lu};
}

template <typename C> using GenStrided = GenWay<false, sizeof(C) == 16 ? 5 : 0>;
using GenLines = GenWay<true, 0>;

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

// d = -1/N / ((i2 + j2) + k2) as ParisPencil.cpp:270-284 sums it, 0 at the zero
// mode, applied to frequency kx of columns kh (and kh + 1).
struct GenFilter {
  int ni, j, kh;
  double j2, ddi, minvN, k2a, k2b;
  __device__ __forceinline__ double at(double i2j2, double k2, int kx, int k) const {
    const double d = recip_pos(i2j2 + k2) * minvN;
    return (kx | j | k) == 0 ? 0.0 : d;
  }
  __device__ __forceinline__ void apply(int kx, double2 &v) const {
    const double id = double(min(kx, ni - kx)) * ddi;
    v = uscale(v, at(id * id + j2, k2a, kx, kh));
  }
  __device__ __forceinline__ void apply(int kx, FPair &v) const {
    const double id = double(min(kx, ni - kx)) * ddi;
    const double s = id * id + j2;
    v.a = cscale(v.a, (float)at(s, k2a, kx, kh));
    v.b = cscale(v.b, (float)at(s, k2b, kx, kh + 1));
  }
};

template <typename C, typename V>
__device__ __forceinline__ void gen_x_tile(const GenPass<C> &a, const GenLane &ln, V *tile, int j, int col0) {
  const int S = a.ax.S;
  const TileLoad<V> ld{tile, a.lu, ln.c};
  gen_dif<GenStrided<C>, false>(a.ax, S - 1, ln, tile, a.lu, ld);
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
      gen_stage<GenStrided<C>, decltype(tag)::value, true, true>(a.ax.st[s], a.ax.tw, ln, tile, a.lu, ld);
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
    gen_dif<GenStrided<C>, KIND == 3>(a.ax, a.ax.S - 1, ln, tile, a.lu, ld);
    gen_y_last<KIND == 3>(a, ln, tile, dst + (long)o * a.nj * a.nhp, kt * W);
  }
}

// ------------------------------------------------------------- z passes
// A block holds `units` columns of line pairs: FP64 unit c is the pair of lines
// (2c, 2c+1); FP32 unit c holds that pair and the pair of lines (2u + 2c,
// 2u + 2c + 1), u the tile's units, so that lanes on neighbouring units read
// lines two pitches apart in both precisions.  Two buffers: the tile and the
// staging area (real lines of pitch lp on one side, spectrum rows of pitch sp
// on the other).  Lines at or past the end are zero in and not stored.
//
// Moves `count` consecutive rows of `bytes` each between HBM (contiguous) and
// staged rows `pitch` bytes apart, one bulk copy per row; bytes, pitch and
// both addresses are multiples of 16.  Lane l of warp 0 takes rows l, l + 32.
__device__ __forceinline__ void rows_in(unsigned char *dst, int pitch, const unsigned char *src, uint32_t bytes,
                                        int count, uint64_t *mbar) {
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) mbar_expect_tx(mbar, bytes * count);
    __syncwarp();
    for (int l = threadIdx.x; l < count; l += 32) bulk_load(dst + l * pitch, src + (long)l * bytes, bytes, mbar);
  }
}
__device__ __forceinline__ void rows_out(unsigned char *dst, uint32_t bytes, const unsigned char *src, int pitch,
                                         int count) {
  if (threadIdx.x < 32) {
    for (int l = threadIdx.x; l < count; l += 32) bulk_store(dst + (long)l * bytes, src + l * pitch, bytes);
    bulk_commit();
    bulk_wait_read();
  }
}

__device__ __forceinline__ bool z_wait(uint64_t *mbar, int *status, int wait_iters) {
  const bool ok = mbar_wait_bounded(mbar, 0, wait_iters);
  if (__syncthreads_or(!ok)) {
    if (threadIdx.x == 0) {
      atomicExch(status, kDevTmaTimeout);
      mbar_wait_bounded(mbar, 0);
    }
    return false;
  }
  return true;
}

// R2C of the real lines (ParisPencil.cpp:152-165).
template <typename T>
__global__ void __launch_bounds__(256, 3)
    k_gen_zfwd(const T *__restrict__ f, typename Cplx<T>::type *spec,
               const __grid_constant__ GenPass<typename Cplx<T>::type> a) {
  using C = typename Cplx<T>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / sizeof(C);      // line pairs per unit
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
  __syncthreads();
  if (a.per_line) {
    rows_in(stage, a.lp * sizeof(T), reinterpret_cast<const unsigned char *>(f + line0 * nk), nk * sizeof(T), nl, &mbar);
  } else if (threadIdx.x == 0) {
    // one contiguous block, rounded up to 16 bytes (the buffer also holds the
    // half spectrum, which is longer)
    const uint32_t bytes = (uint32_t)((size_t)nl * nk * sizeof(T) + 15) & ~15u;
    mbar_expect_tx(&mbar, bytes);
    bulk_load(raw, f + line0 * nk, bytes, &mbar);
  }
  if (threadIdx.x == blockDim.x - 1 && a.l2_ahead > 0) {
    // the lines of the block one resident wave ahead into L2
    const long fl = ((long)blockIdx.x + a.l2_ahead) * lines;
    if (fl < nlines)
      l2_prefetch(f + fl * nk, (uint32_t)((size_t)min((long)lines, nlines - fl) * nk * sizeof(T)) & ~15u);
  }
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  if (nl < lines) {
    for (int q = nl * a.lp + threadIdx.x; q < lines * a.lp; q += blockDim.x) raw[q] = (T)0;
    __syncthreads();
  }
  const GenLane ln = gen_lane(a);
  const T *ra = raw + 2 * ln.c * a.lp;
  const int second = 2 * units * a.lp;   // FP32: the unit's second pair
  auto ld0 = [&](int, int pos, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
    const T *p = ra + pos;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const T *q = p + r * st.m;
      if constexpr (CU == 1) v[r] = mk(q[0], q[a.lp]);
      else v[r] = {mk(q[0], q[a.lp]), mk(q[second], q[second + a.lp])};
    }
  };
  const int S = a.ax.S;
  if (S > 1) {
    gen_dif<GenLines, false>(a.ax, S - 1, ln, tile, a.lu, ld0);
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
  const int second_out = 2 * units * a.sp;
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
  __syncthreads();
  rows_in(stage, a.sp * sizeof(C), reinterpret_cast<const unsigned char *>(spec + line0 * a.nhp), a.nhp * sizeof(C), nl,
          &mbar);
  if (threadIdx.x == blockDim.x - 1 && a.l2_ahead > 0) {
    const long fl = ((long)blockIdx.x + a.l2_ahead) * lines;
    if (fl < nlines)
      l2_prefetch(spec + fl * a.nhp, (uint32_t)((size_t)min((long)lines, nlines - fl) * a.nhp * sizeof(C)));
  }
  if (!z_wait(&mbar, a.status, a.wait_iters)) return;
  // absent lines are zero; the imaginary parts of the zero and Nyquist terms
  // are dropped, as a C2R transform does
  if (nl < lines)
    for (int q = nl * a.sp + threadIdx.x; q < lines * a.sp; q += blockDim.x) rows[q] = mk((T)0, (T)0);
  if ((int)threadIdx.x < nl) {
    rows[threadIdx.x * a.sp].y = (T)0;
    if (nk % 2 == 0) rows[threadIdx.x * a.sp + nk / 2].y = (T)0;
  }
  __syncthreads();
  const GenLane ln = gen_lane(a);
  const C *ra = rows + 2 * ln.c * a.sp;
  const int second = 2 * units * a.sp;
  // Z[k] = A[k] + i B[k] up to n/2, conj A[n-k] + i conj B[n-k] above
  auto ld0 = [&](int, int pos0, const GenStage &st, V *v, auto tag) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int r = 0; r < R; r++) {
      const int pos = pos0 + r * st.m;
      const bool lo = 2 * pos <= nk;
      const C *q = ra + (lo ? pos : nk - pos);
      const T s = lo ? (T)1 : (T)-1;
      auto join = [&](C sa, C sb) { return mk(fma(-s, sb.y, sa.x), fma(s, sa.y, sb.x)); };
      if constexpr (CU == 1) v[r] = join(q[0], q[a.sp]);
      else v[r] = {join(q[0], q[a.sp]), join(q[second], q[second + a.sp])};
    }
  };
  const int S = a.ax.S;
  if (S > 1) {
    gen_dif<GenLines, true>(a.ax, S - 1, ln, tile, a.lu, ld0);
  } else {
    for (int pos = ln.b0; pos < nk; pos += ln.step) ld0(pos, pos, a.ax.st[0], tile + (pos << a.lu) + ln.c, RadixTag<1>{});
    __syncthreads();
  }
  // last stage: real and imaginary parts of points k0 + r n/R to the two real
  // lines of the pair
  const GenStage &s = a.ax.st[S - 1];
  T *out = reinterpret_cast<T *>(stage) + 2 * ln.c * a.lp;
  const int second_out = 2 * units * a.lp;
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
        if constexpr (CU == 1) {
          o[0] = z[r].x;
          o[a.lp] = z[r].y;
        } else {
          o[0] = z[r].a.x;
          o[a.lp] = z[r].a.y;
          o[second_out] = z[r].b.x;
          o[second_out + a.lp] = z[r].b.y;
        }
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
    case 0: return (const void *)k_gen_zfwd<T>;
    case 1: return (const void *)k_gen_strided<T, 1>;
    case 2: return (const void *)k_gen_strided<T, 2>;
    case 3: return (const void *)k_gen_strided<T, 3>;
    default: return (const void *)k_gen_zinv<T>;
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
  const unsigned grid = (unsigned)s.grid;
  switch (kind) {
    case 0: k_gen_zfwd<T><<<grid, s.threads, s.smem, st>>>(static_cast<const T *>(in), static_cast<C *>(out), a); break;
    case 1: k_gen_strided<T, 1><<<grid, s.threads, s.smem, st>>>(*map, static_cast<C *>(out), a); break;
    case 2: k_gen_strided<T, 2><<<grid, s.threads, s.smem, st>>>(*map, static_cast<C *>(out), a); break;
    case 3: k_gen_strided<T, 3><<<grid, s.threads, s.smem, st>>>(*map, static_cast<C *>(out), a); break;
    default: k_gen_zinv<T><<<grid, s.threads, s.smem, st>>>(static_cast<const C *>(in), static_cast<T *>(out), a); break;
  }
  FF_CUDA(cudaGetLastError());
  return FF_OK;
}

#define FF_INSTANTIATE_GEN(T)                                                                               \
  template int gen_prepare<T>(int, size_t);                                                                 \
  template int gen_launch<T>(int, const GenPass<typename Cplx<T>::type> &, const GenShape &, const CUtensorMap *, \
                             const void *, void *, cudaStream_t);

}  // namespace ff
