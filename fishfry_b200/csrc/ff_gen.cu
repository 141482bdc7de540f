// Host side of the passes along axes without a compile-time plan: radix
// splits, device tables and launch shapes (kernels: ff_gen_dev.cuh).

#include "ff_gen.hpp"

#include <cuda_runtime.h>

#include <algorithm>

#include "ff_status.hpp"

namespace ff {

std::vector<int> plan_digit_reversal(int n, const std::vector<int> &radix);

namespace {

// Real operations of one butterfly of radix r on one complex column (additions,
// multiplications and multiply-adds count one each).
int dft_ops(int r) {
  switch (r) {
    case 2: return 4;
    case 3: return 14;
    case 4: return 16;
    case 5: return 36;
    case 6: return 40;
    case 7: return 68;
    case 8: return 56;
    case 9: return 100;
    case 10: return 92;
    default: return 0;
  }
}

// Cost per point of one stage: its two shared-memory accesses and barrier, and
// its arithmetic with (R-1) twiddle products and their powers.
double stage_cost(int r, bool last) {
  const int tw = last ? 0 : 4 * (r - 1) + 4 * (r - 2);
  return 0.40 + (dft_ops(r) + tw + 12.0) / (64.0 * r);
}

void search(int left, std::vector<int> &cur, double cost, const std::vector<int> &lasts, std::vector<int> *best,
            double *best_cost) {
  // a last radix that completes the split
  for (int r : lasts)
    if (left == r) {
      const double c = cost + stage_cost(r, true);
      if (c < *best_cost - 1e-9) {
        *best_cost = c;
        *best = cur;
        best->push_back(r);
      }
    }
  // larger radices first: one order per set of factors
  for (int r = cur.empty() ? kGenMaxRadix : cur.back(); r >= 2; r--) {
    if (left % r != 0 || left == r) continue;
    if ((int)cur.size() + 2 > kGenMaxStages) break;
    cur.push_back(r);
    search(left / r, cur, cost + stage_cost(r, false), lasts, best, best_cost);
    cur.pop_back();
  }
}

}  // namespace

std::vector<int> gen_radices(int n, bool split) {
  if (n <= 1) return {1};
  std::vector<int> lasts;
  for (int r = split ? kGenSplitRadix : kGenMaxRadix; r >= 2; r--) lasts.push_back(r);
  std::vector<int> best, cur;
  double cost = 1e30;
  search(n, cur, 0.0, lasts, &best, &cost);
  return best;
}

std::vector<int> gen_bases(int n, const std::vector<int> &radix) {
  const std::vector<int> rev = plan_digit_reversal(n, radix);
  const int R = radix.back();
  std::vector<int> k0(n / R);
  for (int g = 0; g < n / R; g++) k0[g] = rev[g * R];
  return k0;
}

double gen_cost(int n) {
  const std::vector<int> r = gen_radices(n, false);
  double c = 0.0;
  for (size_t s = 0; s < r.size(); s++) c += stage_cost(r[s], s + 1 == r.size());
  return c;
}

int gen_pad(int n, const std::vector<int> &radix) { return radix.size() > 1 && (n / radix[0]) % 2 == 0 ? 1 : 0; }

int gen_table_size(int n, const std::vector<int> &radix) {
  int L = n, size = 0;
  for (int r : radix) {
    size += (L / r) * ((r + 1) & ~1);
    L /= r;
  }
  return size;
}

void gen_stages(int n, const std::vector<int> &radix, int pad, int threads, int units, int *S, GenStage *st) {
  int L = n, off = 0;
  *S = (int)radix.size();
  const int step = threads / units;
  for (size_t s = 0; s < radix.size(); s++) {
    GenStage &g = st[s];
    g.R = radix[s];
    g.L = L;
    g.m = L / g.R;
    g.nb = n / g.R;
    g.dq = step / g.m;
    g.dr = step % g.m;
    g.inv_m = 1.0f / (float)g.m;
    g.ms = g.m + (s == 0 ? pad : 0);
    g.inv_pb = pad && s > 0 ? (float)L / (float)(n / radix[0]) : 0.0f;
    g.tw = off;
    off += g.m * ((g.R + 1) & ~1);
    L = g.m;
  }
}

void gen_line_stages(int n, const std::vector<int> &radix, int pad, int threads, bool table, int *S, GenStage *st) {
  gen_stages(n, radix, pad, 1, 1, S, st);
  int step = 1;
  for (int s = 0; s < *S; s++) {
    if (table) st[s].tw = step;
    step *= st[s].R;
  }
  st[*S] = GenStage{};
  st[*S].nb = st[*S - 1].nb / 2 + 1;   // frequency bases 0 .. nR/2
  for (int s = 0; s <= *S; s++) {
    st[s].inv_nb = 1.0f / (float)st[s].nb;
    st[s].dq = threads / st[s].nb;
    st[s].dr = threads % st[s].nb;
  }
}

size_t gen_line_smem(int nk, int nhp, int esz, int tile_rows, int W) {
  const int cu = 16 / (2 * esz), units = (W + cu - 1) / cu;
  const size_t lines = (size_t)2 * cu * units;
  const size_t tile = ((size_t)tile_rows * (units | 1) * 16 + 127) & ~size_t(127);
  const size_t stage = std::max(lines * nk * esz + 16, lines * nhp * 2 * esz);
  return tile + ((stage + 127) & ~size_t(127)) + 128;
}

namespace {

size_t r256(size_t b) { return (b + 255) & ~size_t(255); }

// Stage tables [j][r], r < rp = R rounded up to even: exp(-2 pi i j r / L), the
// exponent reduced exactly before FP64 sincospi; one launch for all stages.
struct TableStages {
  int S, total;
  int R[kGenMaxStages], L[kGenMaxStages], off[kGenMaxStages];
};
template <typename C> __global__ void k_gen_twiddles(const TableStages t, C *tw) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < t.total; q += gridDim.x * blockDim.x) {
    int st = t.S - 1;
    while (q < t.off[st]) st--;
    const int rp = (t.R[st] + 1) & ~1, e = q - t.off[st];
    const int j = e / rp, r = e - j * rp;
    double s = 0.0, c = 1.0;
    if (r < t.R[st]) sincospi(2.0 * (double)((long)j * r % t.L[st]) / (double)t.L[st], &s, &c);
    tw[q] = mk((decltype(tw[q].x))c, (decltype(tw[q].x))(-s));
  }
}

}  // namespace

size_t gen_axis_bytes(int n, const std::vector<int> &radix, int esz) {
  return r256((size_t)gen_table_size(n, radix) * 2 * esz);
}

void gen_index(int n, const std::vector<int> &radix, int pad, bool by_frequency, std::vector<int> *out) {
  const std::vector<int> k0 = gen_bases(n, radix);
  if (!by_frequency) {
    *out = k0;
    return;
  }
  const int R = radix.back(), L1 = std::max(1, n / radix[0]);
  out->resize(k0.size());
  for (int g = 0; g < (int)k0.size(); g++) (*out)[k0[g]] = g * R + pad * (g * R / L1);
}

template <typename C> int gen_axis_build(int n, const std::vector<int> &radix, void *mem, const int *idx, GenAxis<C> *ax) {
  if (radix.empty() || radix.size() > (size_t)kGenMaxStages)
    return set_error(FF_ERR_UNSUPPORTED, "no radix split of %d points", n);
  C *tw = static_cast<C *>(mem);
  TableStages t{};
  int L = n;
  for (int r : radix) {
    t.R[t.S] = r;
    t.L[t.S] = L;
    t.off[t.S++] = t.total;
    L /= r;
    t.total += L * ((r + 1) & ~1);
  }
  k_gen_twiddles<<<std::min(256, (t.total + 127) / 128), 128>>>(t, tw);
  FF_CUDA(cudaGetLastError());
  ax->n = n;
  ax->tw = tw;
  ax->idx = idx;
  return FF_OK;
}
template int gen_axis_build<double2>(int, const std::vector<int> &, void *, const int *, GenAxis<double2> *);
template int gen_axis_build<float2>(int, const std::vector<int> &, void *, const int *, GenAxis<float2> *);

namespace {

constexpr size_t kSmSmem = 227 * 1024;

// Smallest v >= lo with v = rem mod step.
int next_congruent(int lo, int rem, int step) { return lo + ((rem - lo) % step + step) % step; }

}  // namespace

// 24 warps on an SM at the tile's shared memory (80 registers a thread).
void gen_pick_threads(GenShape *s) {
  const int blocks = (int)std::max<size_t>(1, std::min<size_t>(8, kSmSmem / (s->smem + 1024)));
  s->threads = std::min(256, std::max(64, 768 / blocks / 32 * 32));
}

void gen_z_shape(GenShape *s, int ni, int nj, int nk, int nhp, int esz, int num_sms, bool lines_kind, size_t limit) {
  const int cu = 16 / (2 * esz);   // line pairs per unit
  const long nlines = (long)ni * nj;
  for (s->units = 8;; s->units /= 2) {
    const int lines = 2 * cu * s->units;
    // pitches that put neighbouring units' lines and rows in different banks
    const bool per_line = (nk * esz) % 16 == 0;
    const int vals = 16 / esz;   // values per 16 bytes
    s->lp = per_line ? next_congruent(nk, std::max(vals, 64 / esz / s->units) % (64 / esz), 64 / esz) : nk;
    const int per = 64 / (2 * esz);
    s->sp = next_congruent(nhp, std::max(cu, per / s->units) % per, per);
    const size_t tile = ((size_t)s->tile_rows * s->units * 16 + 127) & ~size_t(127);
    const size_t stage = std::max((size_t)lines * s->lp * esz + 16, (size_t)lines * s->sp * 2 * esz);
    s->smem = tile + ((stage + 127) & ~size_t(127)) + 128;
    s->grid = (nlines + lines - 1) / lines;
    if (lines_kind) s->smem = gen_line_smem(nk, nhp, esz, s->tile_rows, s->units * cu);
    if (s->units == 1) break;
    if (s->smem <= limit && (s->grid >= num_sms || s->units <= 2)) break;
  }
  gen_pick_threads(s);
}

GenShape gen_shape(int kind, int ni, int nj, int nk, int nhp, int esz, const std::vector<int> &radix, int num_sms) {
  GenShape s{};
  const int cu = 16 / (2 * esz);   // complex columns (or line pairs) per unit
  if (kind == 0 || kind == 4) {
    s.tile_rows = nk + gen_pad(nk, radix) * (radix[0] - 1);
    // many small tiles (up to 40 KB, five or more blocks on an SM) beat fewer
    // large ones for short lines and tie for long ones: 200x180x160 FP32 z
    // 20.9 / 21.5 us against 26.2 / 23.5 at 56 KB, 500^3 FP64 425 / 431 against
    // 443 / 455 at 74 KB
    gen_z_shape(&s, ni, nj, nk, nhp, esz, num_sms, esz == 4, 40 * 1024);
    return s;
  }
  const int n = kind == 2 ? ni : nj;
  const int nh = nk / 2 + 1;
  // 128-byte rows while three tiles fit an SM (up to 590 points; 64-byte rows
  // there measured 2-5 % slower: 384^3 FP64 y 184 against 180 us, FP32 111
  // against 106), else 64-byte rows, which keep four or more 24 KB to 75 KB tiles on
  // an SM where 128-byte rows leave two (640x640x320 FP64 y 430 us; 698 before
  // with 128-byte rows), and 32-byte ones for lines whose tile would not fit
  for (s.units = 8;; s.units /= 2) {
    // equal TMA boxes of at most 256 rows that start on 128 bytes of shared
    // memory; the last one may reach past the line (zero fill, clipped stores)
    const int align = 8 / s.units;
    for (int boxes = (n + 255) / 256;; boxes++) {
      s.box_rows = ((n + boxes - 1) / boxes + align - 1) / align * align;
      if (s.box_rows <= 256) break;
    }
    s.smem = (size_t)((n + s.box_rows - 1) / s.box_rows * s.box_rows) * s.units * 16 + 128;
    const int w = s.units * cu;
    s.grid = (long)(kind == 2 ? nj : ni) * ((nh + w - 1) / w);
    if (s.units == 2) break;
    if (s.units == 8 ? s.smem <= 74 * 1024 && s.grid >= num_sms : s.smem <= kSmSmem - 1024) break;
  }
  gen_pick_threads(&s);
  return s;
}

}  // namespace ff
