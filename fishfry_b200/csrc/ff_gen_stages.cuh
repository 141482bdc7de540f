// Shared-memory stages for plans read at run time, on 16-byte units: the engine
// of the generic passes (ff_gen_dev.cuh) and of the Bluestein passes
// (ff_bluestein.cu).
//
// Every tile is point-major in units of 16 bytes: [row][unit], a unit being one
// FP64 or two adjacent FP32 complex columns (z passes: one FP64 line pair or
// two FP32 ones, as complex lines), so both precisions run the same code on
// 16-byte shared-memory accesses.  Threads take units fastest: a thread keeps
// its unit, and walks butterflies b0, b0 + step, ... of that column.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <type_traits>

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

// m + s u and m - s u.  FP32 as two multiply-adds, which round once each (the
// negated u costs what the product did: FFMA2 takes no negated operands, and a
// second constant of either sign took registers that the last stages spilled:
// 480x400x360 FP32 y 139 / 137 -> 145 / 150 us); FP64 as a product, a sum and a
// difference (multiply-adds there lengthen the chain: 500^3 z 452 / 459 -> 469 / 475).
__device__ __forceinline__ void upm(double2 m, double2 u, double s, double2 &p, double2 &q) {
  const double2 w = uscale(u, s);
  p = uadd(m, w);
  q = usub(m, w);
}
__device__ __forceinline__ void upm(FPair m, FPair u, float s, FPair &p, FPair &q) {
  p = ufma(u, s, m);
  q = ufma(uscale(u, -1.0f), s, m);
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
  const V u = umul_wi<INV>(usub(v1, v2));
  const V m = ufma(t, (T)-0.5, v0);
  v0 = uadd(v0, t);
  upm(m, u, (T)FF_SQRT3_2, v1, v2);
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
    const V o1 = uadd(v[3], umul_wi<INV>(v[3]));   // times sqrt 2
    const V o2 = umul_wi<INV>(v[5]);
    const V o3 = usub(umul_wi<INV>(v[7]), v[7]);   // times sqrt 2
    const V e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = uadd(e0, o0);
    v[4] = usub(e0, o0);
    upm(e1, o1, h, v[1], v[5]);
    v[2] = uadd(e2, o2);
    v[6] = usub(e2, o2);
    upm(e3, o3, h, v[3], v[7]);
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
template <int R, bool CONJ, typename WH>
__device__ __forceinline__ void gen_powers(double2 *v, double2 w1, WH &&half) {
  double2 w = w1;
  if constexpr (R < 6) {
#pragma unroll
    for (int r = 1; r < R; r++) {
      v[r] = ucmul<CONJ>(v[r], w);
      if (r + 1 < R) w = cmul(w, w1);
    }
  } else {
    constexpr int H = (R + 1) / 2;
    const double2 wh = half();
    v[H] = ucmul<CONJ>(v[H], wh);
#pragma unroll
    for (int r = 1; r < H; r++) {
      v[r] = ucmul<CONJ>(v[r], w);
      if (H + r < R) v[H + r] = ucmul<CONJ>(v[H + r], cmul(wh, w));
      if (r + 1 < H) w = cmul(w, w1);
    }
  }
}
template <int R, bool CONJ>
__device__ __forceinline__ void gen_twiddle(double2 *v, const double2 *__restrict__ t) {
  gen_powers<R, CONJ>(v, __ldg(t + 1), [&] { return __ldg(t + (R + 1) / 2); });
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

// Twiddles of the packed per-stage tables (GenAxis) and of an axis's plain table
// (AxisDev: entry q = exp(-2 pi i q / n); GenStage::tw is then the step n / L).
template <typename C> struct PackedTw {
  const C *tw;
  template <int R, bool CONJ, typename V> __device__ __forceinline__ void apply(V *v, const GenStage &s, int j) const {
    gen_twiddle<R, CONJ>(v, tw + s.tw + j * ((R + 1) & ~1));
  }
};
template <typename C> struct AxisTw;
template <> struct AxisTw<double2> {
  const double2 *tw;
  template <int R, bool CONJ> __device__ __forceinline__ void apply(double2 *v, const GenStage &s, int j) const {
    gen_powers<R, CONJ>(v, __ldg(tw + j * s.tw), [&] { return __ldg(tw + j * ((R + 1) / 2) * s.tw); });
  }
};
template <> struct AxisTw<float2> {
  const float2 *tw;
  template <int R, bool CONJ> __device__ __forceinline__ void apply(FPair *v, const GenStage &s, int j) const {
#pragma unroll
    for (int r = 1; r < R; r++) v[r] = ucmul<CONJ>(v[r], __ldg(tw + j * r * s.tw));
  }
};

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

// Stores to the tile.
template <typename V> struct TilePut {
  V *tile;
  int lu, c;
  template <int R>
  __device__ __forceinline__ void operator()(int row, int, const GenStage &s, const V *v, RadixTag<R>) const {
    V *p = tile + (row << lu) + c;
    const int step = s.ms << lu;
#pragma unroll
    for (int r = 0; r < R; r++) p[r * step] = v[r];
  }
};

// A stage: ld(row, pos, s, v) fills a butterfly's R points (positions pos + r m,
// tile rows row + r ms), put(row, pos, s, v) takes the result.  The thread walks
// its butterflies b0, b0 + step, ... of the column.
template <typename WAY, int R, bool INV, bool DIT, typename V, typename TW, typename LD, typename ST>
__device__ __forceinline__ void gen_stage(const GenStage &s, const TW &tw, const GenLane &ln, LD &&ld, ST &&put) {
  constexpr RadixTag<R> tag{};
  // tile to tile: one pointer and stride for both sides
  constexpr bool kPut = std::is_same<std::decay_t<ST>, TilePut<V>>::value;
  constexpr bool kLoad = kPut && std::is_same<std::decay_t<LD>, TileLoad<V>>::value;
  int stride = 0;
  if constexpr (kPut) stride = (WAY::kPad ? s.ms : s.m) << put.lu;
  auto at = [&](int row) -> V * {
    if constexpr (kPut) return put.tile + (row << put.lu) + put.c;
    else return nullptr;
  };
  auto load = [&](int row, int pos, V *p, V *v) {
    if constexpr (kLoad) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = p[r * stride];
    } else {
      ld(row, pos, s, v, tag);
    }
  };
  auto store = [&](int row, int pos, V *p, const V *v) {
    if constexpr (kPut) {
#pragma unroll
      for (int r = 0; r < R; r++) p[r * stride] = v[r];
    } else {
      put(row, pos, s, v, tag);
    }
  };
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
    if (DIT && s.m > 1) tw.template apply<R, INV>(v, s, jj);
    UDft<R, INV, V>::run(v);
    if (!DIT && s.m > 1) tw.template apply<R, INV>(v, s, jj);
  };
  int b = ln.b0;
  if constexpr (R <= WAY::kPair) {
    for (; b + ln.step < s.nb; b += 2 * ln.step) {
      const int j1 = j, pos1 = q * s.L + j, row1 = row_of(pos1);
      advance();
      const int pos2 = q * s.L + j, row2 = row_of(pos2);
      V *p1 = at(row1), *p2 = at(row2);
      V v[R], w[R];
      load(row1, pos1, p1, v);
      load(row2, pos2, p2, w);
      work(v, j1);
      work(w, j);
      store(row1, pos1, p1, v);
      store(row2, pos2, p2, w);
      advance();
    }
  }
  for (; b < s.nb; b += ln.step) {
    const int pos = q * s.L + j, row = row_of(pos);
    V *p = at(row);
    V v[R];
    load(row, pos, p, v);
    work(v, j);
    store(row, pos, p, v);
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

// DIF stages 0 .. s1-1 in the tile, each followed by a barrier; the first reads
// through ld0.
template <typename WAY, bool INV, typename V, typename TW, typename LD0>
__device__ __forceinline__ void gen_dif(const GenStage *st, int s1, const TW &tw, const GenLane &ln, V *tile, int lu,
                                        LD0 &&ld0) {
  const TileLoad<V> ld{tile, lu, ln.c};
  const TilePut<V> put{tile, lu, ln.c};
  for (int s = 0; s < s1; s++) {
    with_gen_radix(st[s].R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      if constexpr (std::is_same<std::decay_t<LD0>, TileLoad<V>>::value) {
        gen_stage<WAY, R, INV, false, V>(st[s], tw, ln, ld, put);
      } else {
        if (s == 0) gen_stage<WAY, R, INV, false, V>(st[s], tw, ln, ld0, put);
        else gen_stage<WAY, R, INV, false, V>(st[s], tw, ln, ld, put);
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

// ------------------------------------------------------- rows of the z passes
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

// A tile's real lines line0 .. line0 + nl - 1 into staged lines of pitch lp: one
// copy per line, or one contiguous block rounded up to 16 bytes (the buffer
// also holds the half spectrum, which is longer).
template <typename C, typename T>
__device__ __forceinline__ void lines_in(const GenPass<C> &a, T *raw, const T *f, long line0, int nl, uint64_t *mbar) {
  if (a.per_line) {
    rows_in(reinterpret_cast<unsigned char *>(raw), a.lp * sizeof(T),
            reinterpret_cast<const unsigned char *>(f + line0 * a.nk), a.nk * sizeof(T), nl, mbar);
  } else if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)((size_t)nl * a.nk * sizeof(T) + 15) & ~15u;
    mbar_expect_tx(mbar, bytes);
    bulk_load(raw, f + line0 * a.nk, bytes, mbar);
  }
}

// Staged spectrum rows before a C2R: absent lines are zero, and the imaginary
// parts of the zero and Nyquist terms are dropped, as a C2R transform does.
template <typename C>
__device__ __forceinline__ void z_rows_real_ends(const GenPass<C> &a, C *rows, int nl, int lines) {
  using T = typename Real<C>::type;
  if (nl < lines)
    for (int q = nl * a.sp + threadIdx.x; q < lines * a.sp; q += blockDim.x) rows[q] = mk((T)0, (T)0);
  if ((int)threadIdx.x < nl) {
    rows[threadIdx.x * a.sp].y = (T)0;
    if (a.nk % 2 == 0) rows[threadIdx.x * a.sp + a.nk / 2].y = (T)0;
  }
}

// Lines of a unit in staged memory: a pair's second line lies `pitch` behind its
// first; FP32's second pair `second` behind the first pair.
// Two real lines at q as one complex line, and back.
template <typename V, typename T> __device__ __forceinline__ V unit_of(const T *q, int pitch, int second) {
  if constexpr (sizeof(T) == 8) return mk(q[0], q[pitch]);
  else return {mk(q[0], q[pitch]), mk(q[second], q[second + pitch])};
}
template <typename V, typename T> __device__ __forceinline__ void unit_put(T *q, int pitch, int second, V v) {
  if constexpr (sizeof(T) == 8) {
    q[0] = v.x;
    q[pitch] = v.y;
  } else {
    q[0] = v.a.x;
    q[pitch] = v.a.y;
    q[second] = v.b.x;
    q[second + pitch] = v.b.y;
  }
}

// A[k] = (Z[k] + conj Z[n-k]) / 2 and B[k] = (Z[k] - conj Z[n-k]) / (2i), p = Z[k],
// q = Z[n-k], to the rows at o of the unit's lines (ParisPencil.cpp:152-165).
template <typename V, typename C> __device__ __forceinline__ void unit_split(C *o, int pitch, int second, V p, V q) {
  using T = typename Real<C>::type;
  const T h = (T)0.5;
  auto emit = [&](C *r, C zp, C zq) {
    r[0] = mk(h * (zp.x + zq.x), h * (zp.y - zq.y));
    r[pitch] = mk(h * (zp.y + zq.y), h * (zq.x - zp.x));
  };
  if constexpr (sizeof(C) == 16) {
    emit(o, p, q);
  } else {
    emit(o, p.a, q.a);
    emit(o + second, p.b, q.b);
  }
}

// Point pos of the Hermitian extension of a unit's rows (row a of a pair at q, row
// b a pitch behind): Z[k] = A[k] + i B[k] up to n/2, conj A[n-k] + i conj B[n-k]
// above (ParisPencil.cpp:368-380).
template <typename V, typename C>
__device__ __forceinline__ V unit_extend(const C *ra, int pitch, int second, int nk, int pos) {
  using T = typename Real<C>::type;
  const bool lo = 2 * pos <= nk;
  const C *q = ra + (lo ? pos : nk - pos);
  const T s = lo ? (T)1 : (T)-1;
  auto join = [&](C sa, C sb) { return mk(fma(-s, sb.y, sa.x), fma(s, sa.y, sb.x)); };
  if constexpr (sizeof(C) == 16) return join(q[0], q[pitch]);
  else return {join(q[0], q[pitch]), join(q[second], q[second + pitch])};
}

}  // namespace ff
