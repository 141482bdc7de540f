// z tiles with butterflies fastest: the FP32 z passes of lengths without a
// compile-time plan, and the batched z passes of such lengths (any number of
// line pairs per tile).
#pragma once

#include "ff_gen_stages.cuh"

namespace ff {

// The last radix of a z tile here: at most kGenSplitRadix in the packed plans, 8
// too in an axis's own radix order (batched passes).
template <typename F> __device__ __forceinline__ void with_line_radix(int r, F &&f) {
  if (r == 8) f(RadixTag<8>{});
  else with_split_radix(r, f);
}

// ------------------------------------------------------------ z tiles
// A z tile is `units` columns of line pairs (FP64 unit c: the pair of lines 2c,
// 2c+1; FP32: that pair and the pair of lines 2u + 2c, 2u + 2c + 1, u the units)
// by the line's points, rows `units | 1` units long: an odd number, so that
// lanes on consecutive rows are in different banks.  Threads take butterflies
// fastest: the staged lines are then read and written along the line, as they
// lie in HBM, and need no padding, so a tile moves by one bulk copy each way.
template <typename V> struct LineUnits {
  V *tile;
  int pitch;   // units | 1
  int units;
};

// Items t, t + threads, ... of `s` over all columns: f(column, butterfly).
template <typename F> __device__ __forceinline__ void line_items(const GenStage &s, int units, F &&f) {
  int c = __float2int_rz(((float)threadIdx.x + 0.5f) * s.inv_nb);
  int b = (int)threadIdx.x - c * s.nb;
  while (c < units) {
    f(c, b);
    c += s.dq;
    b += s.dr;
    if (b >= s.nb) { b -= s.nb; c++; }
  }
}

// A stage of a z tile: ld(c, pos, s, v) fills a butterfly's R points
// (positions pos + r m; null: from the tile), put(c, pos, s, v) takes the
// result (null: to the tile).
struct InTile {};
template <int R, bool INV, bool DIT, typename V, typename TW, typename LD, typename ST>
__device__ __forceinline__ void line_stage(const GenStage &s, const TW &tw, const LineUnits<V> &t, LD &&ld, ST &&put) {
  constexpr bool kLoad = std::is_same<std::decay_t<LD>, InTile>::value;
  constexpr bool kPut = std::is_same<std::decay_t<ST>, InTile>::value;
  const int stride = s.ms * t.pitch;
  line_items(s, t.units, [&](int c, int b) {
    const int q = __float2int_rz(((float)b + 0.5f) * s.inv_m);
    const int j = b - q * s.m;
    const int pos = q * s.L + j;
    V *p = t.tile + (pos + __float2int_rz(((float)q + 0.5f) * s.inv_pb)) * t.pitch + c;
    V v[R];
    if constexpr (kLoad) {
#pragma unroll
      for (int r = 0; r < R; r++) v[r] = p[r * stride];
    } else {
      ld(c, pos, s, v, RadixTag<R>{});
    }
    if (DIT && s.m > 1) tw.template apply<R, INV>(v, s, j);
    UDft<R, INV, V>::run(v);
    if (!DIT && s.m > 1) tw.template apply<R, INV>(v, s, j);
    if constexpr (kPut) {
#pragma unroll
      for (int r = 0; r < R; r++) p[r * stride] = v[r];
    } else {
      put(c, pos, s, v, RadixTag<R>{});
    }
  });
}

// DIF stages 0 .. s1-1, each followed by a barrier; the first reads through ld0.
template <bool INV, typename V, typename TW, typename LD0>
__device__ __forceinline__ void line_dif(const GenStage *st, int s1, const TW &tw, const LineUnits<V> &t, LD0 &&ld0) {
  for (int s = 0; s < s1; s++) {
    with_gen_radix(st[s].R, [&](auto tag) {
      constexpr int R = decltype(tag)::value;
      if (s == 0) line_stage<R, INV, false, V>(st[s], tw, t, ld0, InTile{});
      else line_stage<R, INV, false, V>(st[s], tw, t, InTile{}, InTile{});
    });
    __syncthreads();
  }
}

// The lines of unit c of a tile.  The same values as unit_of and the like
// (ff_gen_stages.cuh) form at a lane's fixed unit, addressed from the tile's
// start: written in terms of those the kernels here lost (480x400x360 FP32 z
// inverse 144 -> 153 to 163 us, 48 grids of ragged lengths FP64 999 -> 1009).
// Point pos of unit c of staged real lines as complex values.
template <typename V, typename T> __device__ __forceinline__ V line_pair(const T *raw, int nk, int units, int c, int pos) {
  const T *q = raw + 2 * c * nk + pos;
  if constexpr (sizeof(T) == 8) {
    return mk(q[0], q[nk]);
  } else {
    const T *q2 = q + 2 * units * nk;
    return {mk(q[0], q[nk]), mk(q2[0], q2[nk])};
  }
}
// And back: real and imaginary parts to the two lines of a pair.
template <typename V, typename T>
__device__ __forceinline__ void line_pair_put(T *raw, int nk, int units, int c, int pos, V v) {
  T *q = raw + 2 * c * nk + pos;
  if constexpr (sizeof(T) == 8) {
    q[0] = v.x;
    q[nk] = v.y;
  } else {
    T *q2 = q + 2 * units * nk;
    q[0] = v.a.x;
    q[nk] = v.a.y;
    q2[0] = v.b.x;
    q2[nk] = v.b.y;
  }
}

// A[k] = (Z[k] + conj Z[n-k]) / 2 and B[k] = (Z[k] - conj Z[n-k]) / (2i), p = Z[k],
// q = Z[n-k], to the staged rows of unit c's lines (ParisPencil.cpp:152-165).
template <typename V, typename C>
__device__ __forceinline__ void line_split(C *rows, int nhp, int units, int c, int k, V p, V q) {
  using T = typename Real<C>::type;
  const T h = (T)0.5;
  auto emit = [&](C *o, C zp, C zq) {
    o[0] = mk(h * (zp.x + zq.x), h * (zp.y - zq.y));
    o[nhp] = mk(h * (zp.y + zq.y), h * (zq.x - zp.x));
  };
  C *o = rows + 2 * c * nhp + k;
  if constexpr (sizeof(C) == 16) {
    emit(o, p, q);
  } else {
    emit(o, p.a, q.a);
    emit(o + 2 * units * nhp, p.b, q.b);
  }
}

// Point pos of the Hermitian extension of unit c's staged rows: Z[k] = A[k] + i
// B[k] up to n/2, conj A[n-k] + i conj B[n-k] above (ParisPencil.cpp:368-380).
template <typename V, typename C>
__device__ __forceinline__ V line_extend(const C *rows, int nk, int nhp, int units, int c, int pos) {
  using T = typename Real<C>::type;
  const bool lo = 2 * pos <= nk;
  const C *q = rows + 2 * c * nhp + (lo ? pos : nk - pos);
  const T s = lo ? (T)1 : (T)-1;
  auto join = [&](C sa, C sb) { return mk(fma(-s, sb.y, sa.x), fma(s, sa.y, sb.x)); };
  if constexpr (sizeof(C) == 16) {
    return join(q[0], q[nhp]);
  } else {
    const C *q2 = q + 2 * units * nhp;
    return {join(q[0], q[nhp]), join(q2[0], q2[nhp])};
  }
}

// The staged rows before that: absent lines are zero, and the imaginary parts
// of the zero and Nyquist terms are dropped, as a C2R transform does.
template <typename C>
__device__ __forceinline__ void line_rows_fix(C *rows, int nk, int nhp, int nl, int lines) {
  using T = typename Real<C>::type;
  for (int q = nl * nhp + threadIdx.x; q < lines * nhp; q += blockDim.x) rows[q] = mk((T)0, (T)0);
  for (int l = threadIdx.x; l < nl; l += blockDim.x) {
    rows[l * nhp].y = (T)0;
    if (nk % 2 == 0) rows[l * nhp + nk / 2].y = (T)0;
  }
}

// The z tile of a block: buffers and lines.
template <typename C> struct LineTileOf {
  using T = typename Real<C>::type;
  using V = typename Unit<C>::type;
  LineUnits<V> t;
  T *raw;         // staged real lines, nk values each
  C *rows;        // the same memory as staged spectrum rows, nhp values each
  int nk, nhp;
  int lines, nl;  // lines of the tile, and how many of them there are
  long line0;
};
// Tile `tile` of W line pairs (FP32: an odd W leaves the last unit's second pair
// absent); rows: its padded rows.
template <typename C>
__device__ __forceinline__ LineTileOf<C> line_tile(int nk, int nhp, long nlines, int W, int rows, long tile,
                                                   unsigned char *sm) {
  using T = typename Real<C>::type;
  using V = typename Unit<C>::type;
  constexpr int CU = 16 / sizeof(C);
  const int units = (W + CU - 1) / CU;
  LineTileOf<C> b;
  b.t = {reinterpret_cast<V *>(sm), units | 1, units};
  unsigned char *stage = reinterpret_cast<unsigned char *>(b.t.tile + (((rows * b.t.pitch) + 7) & ~7));
  b.raw = reinterpret_cast<T *>(stage);
  b.rows = reinterpret_cast<C *>(stage);
  b.nk = nk;
  b.nhp = nhp;
  b.lines = 2 * CU * units;
  b.line0 = tile * (2 * W);
  b.nl = (int)min((long)(2 * W), nlines - b.line0);
  return b;
}

// R2C of the staged real lines into the staged spectrum rows (ParisPencil.cpp:152-165).
// first[k0]: tile row of the last-stage group of frequency base k0, through
// row_of.  Ends without a barrier.
template <typename C, typename TW, typename ROW>
__device__ __forceinline__ void line_forward(const LineTileOf<C> &b, const GenStage *st, int S, const TW &tw,
                                             const ROW &row_of) {
  using T = typename Real<C>::type;
  using V = typename Unit<C>::type;
  const int nk = b.nk, units = b.t.units;
  if (b.nl < b.lines) {
    for (int q = b.nl * nk + threadIdx.x; q < b.lines * nk; q += blockDim.x) b.raw[q] = (T)0;
    __syncthreads();
  }
  if (S > 1) {
    line_dif<false>(st, S - 1, tw, b.t, [&](int c, int pos, const GenStage &s, V *v, auto tag) {
#pragma unroll
      for (int r = 0; r < decltype(tag)::value; r++) v[r] = line_pair<V>(b.raw, nk, units, c, pos + r * s.m);
    });
  } else {
    // one stage: the split reads the tile
    for (int q = threadIdx.x; q < units * nk; q += blockDim.x)
      b.t.tile[q % nk * b.t.pitch + q / nk] = line_pair<V>(b.raw, nk, units, q / nk, q % nk);
    __syncthreads();
  }
  // Last stage and split: the groups of bases k0 and nR - k0 (nR = n/R) hold
  // Z[k0 + r nR] and, at R-1-r, Z[n - (k0 + r nR)]; base 0 pairs with itself
  // shifted by one and nR/2 with itself (their pairs come out twice, the same
  // values).
  const int nR = st[S - 1].nb;
  with_line_radix(st[S - 1].R, [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    line_items(st[S], units, [&](int c, int k0) {
      V z1[R], z2[R];
      const V *p1 = b.t.tile + row_of(k0) * b.t.pitch + c;
#pragma unroll
      for (int r = 0; r < R; r++) z1[r] = p1[r * b.t.pitch];
      UDft<R, false, V>::run(z1);
      if (k0 > 0) {
        const V *p2 = b.t.tile + row_of(nR - k0) * b.t.pitch + c;
#pragma unroll
        for (int r = 0; r < R; r++) z2[r] = p2[r * b.t.pitch];
        UDft<R, false, V>::run(z2);
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) z2[r] = z1[(r + 1) % R];
      }
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (2 * r < R) line_split(b.rows, b.nhp, units, c, k0 + r * nR, z1[r], z2[R - 1 - r]);
        else line_split(b.rows, b.nhp, units, c, nk - k0 - r * nR, z2[R - 1 - r], z1[r]);
      }
    });
  });
}

// C2R of the staged spectrum rows into the staged real lines (ParisPencil.cpp:368-380).
template <typename C, typename TW, typename ROW>
__device__ __forceinline__ void line_inverse(const LineTileOf<C> &b, const GenStage *st, int S, const TW &tw,
                                             const ROW &row_of) {
  using V = typename Unit<C>::type;
  const int nk = b.nk, units = b.t.units;
  line_rows_fix(b.rows, nk, b.nhp, b.nl, b.lines);
  __syncthreads();
  if (S > 1) {
    line_dif<true>(st, S - 1, tw, b.t, [&](int c, int pos, const GenStage &s, V *v, auto tag) {
#pragma unroll
      for (int r = 0; r < decltype(tag)::value; r++)
        v[r] = line_extend<V>(b.rows, nk, b.nhp, units, c, pos + r * s.m);
    });
  } else {
    for (int q = threadIdx.x; q < units * nk; q += blockDim.x)
      b.t.tile[q % nk * b.t.pitch + q / nk] = line_extend<V>(b.rows, nk, b.nhp, units, q / nk, q % nk);
    __syncthreads();
  }
  // last stage: points k0 + r n/R to the real lines
  const GenStage &s = st[S - 1];
  with_line_radix(s.R, [&](auto tag) {
    constexpr int R = decltype(tag)::value;
    line_items(s, units, [&](int c, int k0) {
      V z[R];
      const V *p = b.t.tile + row_of(k0) * b.t.pitch + c;
#pragma unroll
      for (int r = 0; r < R; r++) z[r] = p[r * b.t.pitch];
      UDft<R, true, V>::run(z);
#pragma unroll
      for (int r = 0; r < R; r++) line_pair_put(b.raw, nk, units, c, k0 + r * s.nb, z[r]);
    });
  });
}

}  // namespace ff
