// The batched form: many independent grids of uneven sizes solved by five
// launches (one per pass) captured once in a CUDA graph, with
// tile shapes picked by a measuring autotuner.  Each grid's solve is the
// single-grid algorithm (ParisPencil.cpp:95-425 restated as five passes).
//
// Host side: axis tables shared by all grids of one length, the grid
// descriptors, the per-pass work lists (prefix sums of tiles over grids), the
// graph, and the tuner.  The kernels are in ff_batch_dev.cuh.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "ff_batch.hpp"
#include "ff_status.hpp"
#include "ff_tiles.cuh"

namespace ff {

// Shared with the single-grid plan (ff_solve.cu).
std::vector<int> plan_factor_radices(int n);
std::vector<int> plan_digit_reversal(int n, const std::vector<int> &radix);

namespace {

// Tuned shapes, process-wide: (precision, pass kind, axis length) -> shape.
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int>, TileShape> g_tuned;

int axis_of_kind(int kind) { return kind == 0 || kind == 4 ? 2 : kind == 2 ? 0 : 1; }

}  // namespace
}  // namespace ff

using namespace ff;

struct ff_batch {
  int count = 0;
  int precision = FF_FP64;
  int device = 0;
  int num_sms = 0;
  size_t csz = 16;
  std::vector<BatchGridHost> grids;
  std::vector<size_t> bytes;
  void *dmem = nullptr;          // axis tables, status, descriptors, work lists
  size_t dmem_size = 0;
  int *status = nullptr;
  void *desc = nullptr;          // device grid descriptors
  size_t desc_size = 0;
  unsigned char *desc_host = nullptr;   // pinned image of the descriptors
  CUtensorMap *maps = nullptr;          // device: two tensor maps per grid (y, x boxes of its potential)
  CUtensorMap *maps_host = nullptr;     // pinned image
  int *entries[5] = {};
  int *starts[5] = {};
  int ntiles[5] = {};
  int ahead[5] = {};             // blocks resident at once
  size_t smem[5] = {};
  bool desc_dirty = true;
  // axis tables by (length, radix order); default orders live in dmem, other
  // orders (from the tuner) in their own allocations
  std::map<std::pair<int, int>, std::pair<AxisDev<double2>, AxisDev<float2>>> tables;
  std::vector<void *> extra;
  cudaStream_t cap = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t ev[6] = {};
  // Grids the batch kernels cannot hold (an axis with a prime factor above 7,
  // or longer than their tiles) are solved by their own single-grid plans
  // (Bluestein passes where needed) after the batched launches, on the same
  // stream.  where[u] of caller index u: >= 0 the index among the batched
  // grids, < 0 side grid -where[u]-1.
  int user_count = 0;
  std::vector<int> where;
  std::vector<ff_plan *> side;
  std::vector<size_t> side_bytes;
  cudaEvent_t side_ev[2] = {};
};

namespace ff {
namespace {

size_t desc_size(int precision) {
  return precision == FF_FP64 ? batch_desc_size<double>() : batch_desc_size<float>();
}

void desc_fill(int precision, void *dst, const BatchGridHost &g) {
  if (precision == FF_FP64) batch_desc_fill<double>(dst, g);
  else batch_desc_fill<float>(dst, g);
}

int pass_prepare(int precision, int kind, size_t smem, int *per_sm) {
  return precision == FF_FP64 ? batch_pass_prepare<double>(kind, smem, per_sm)
                              : batch_pass_prepare<float>(kind, smem, per_sm);
}

int pass_launch(const ff_batch *b, int kind, cudaStream_t st) {
  const BatchWork wl{b->entries[kind], b->starts[kind], b->count, b->ahead[kind]};
  return b->precision == FF_FP64
             ? batch_pass_launch<double>(kind, b->desc, b->maps, wl, b->ntiles[kind], b->smem[kind], st)
             : batch_pass_launch<float>(kind, b->desc, b->maps, wl, b->ntiles[kind], b->smem[kind], st);
}

}  // namespace

int batch_axis_len(const BatchGridHost &g, int kind) { return g.n[axis_of_kind(kind)]; }

int batch_tiles_of(const BatchGridHost &g, int kind) {
  const TileShape &s = g.shape[kind];
  if (kind == 0 || kind == 4) {
    const long npairs = ((long)g.n[0] * g.n[1] + 1) / 2;
    return (int)((npairs + s.W - 1) / s.W);
  }
  const long planes = kind == 2 ? g.n[1] : g.n[0];
  if (s.tma) return (int)(planes * ((g.nh + s.W - 1) / s.W));
  // FP32 columns go in pairs: rows count their padding column
  const long ncols = planes * g.nhp;
  return (int)((ncols + s.W - 1) / s.W);
}

size_t batch_shape_smem(int precision, const BatchGridHost &g, int kind, const TileShape &s) {
  return batch_tile_smem(kind, batch_axis_len(g, kind), g.n[2], g.nhp, s.W, s.ct, precision == FF_FP64 ? 16 : 8);
}

// z passes of a runtime length may move line blocks by bulk copies when the
// lines are 16-byte multiples and the plan has two or more stages (lines of one
// stage, up to 8 points, are left to the threads).
bool batch_z_bulk_ok(int precision, int nk) {
  return ((size_t)nk * (precision == FF_FP64 ? 8 : 4)) % 16 == 0 && plan_stages(nk) >= 2;
}

bool batch_shape_valid(int precision, const BatchGridHost &g, int kind, const TileShape &s) {
  if (s.W < 1) return false;
  if (s.order != 0 && (s.ct || kind > 2 || batch_radix_order(batch_axis_len(g, kind), s.order).empty())) return false;
  if (s.ct && !batch_special_n(batch_axis_len(g, kind))) return false;
  if (kind != 0 && kind != 4) {
    const int w1 = 128 / (precision == FF_FP64 ? 16 : 8);
    if (s.W != w1 && s.W != 2 * w1 && s.W != 4 * w1) return false;
    if (s.tma && s.W != w1) return false;
  } else if (s.tma && !batch_z_bulk_ok(precision, g.n[2])) {
    return false;
  }
  return batch_shape_smem(precision, g, kind, s) <= batch_budget(kind);
}

// Default shape: strided tiles of about 4096 points (256 threads) and z tiles
// of about 2048 (128 threads), a few butterfly items per thread and stage,
// within the pass's shared-memory budget; compile-time tiles where the
// length has them.
TileShape batch_default_shape(int precision, const BatchGridHost &g, int kind) {
  const int n = batch_axis_len(g, kind);
  TileShape s{1, batch_special_n(n) ? 1 : 0, 0};
  if (kind == 0 || kind == 4) {
    const long npairs = ((long)g.n[0] * g.n[1] + 1) / 2;
    // about 2048 points per tile (two butterfly items per thread of the
    // 128-thread z blocks); longer lines take up to 32 KB of line pairs (at
    // most 8), as the single-grid z passes do, so that each block moves
    // enough bytes per copy
    const size_t csz = precision == FF_FP64 ? 16 : 8;
    const int align = csz == 16 ? 8 : 16;
    const size_t per_pair = 2 * (size_t)((g.n[2] + align - 1) / align * align) * csz;
    // FP32 tiles of compile-time lengths: twice that (their lines are half as
    // long in bytes; 60 grids of 32 to 128 points: z passes 110 / 110 -> 94 / 92 us)
    int W = std::max(1, (precision == FF_FP32 && s.ct ? 2048 : 1024) / std::max(1, g.n[2]));
    W = std::max(W, (int)std::max<size_t>(1, std::min<size_t>(8, (32 * 1024) / per_pair)));
    W = (int)std::min<long>(W, npairs);
    while (W > 1 && !batch_shape_valid(precision, g, kind, TileShape{W, s.ct, 0})) W--;
    s.W = W;
    // runtime lengths: bulk-copied line blocks where the lines allow them
    // (compile-time lengths always use them)
    s.tma = !s.ct && batch_z_bulk_ok(precision, g.n[2]) ? 1 : 0;
    return s;
  }
  const int w1 = 128 / (precision == FF_FP64 ? 16 : 8);
  // long lines with many columns per plane: one-plane tiles by TMA, as the
  // single-grid passes
  if (n >= 256 && g.nh >= 4 * w1) {
    s.W = w1;
    s.tma = 1;
    return s;
  }
  int W = w1;
  for (int m = 4; m >= 1; m /= 2) {
    const TileShape t{m * w1, s.ct, 0};
    if (m * w1 * n <= 4096 && batch_shape_valid(precision, g, kind, t)) {
      W = m * w1;
      break;
    }
  }
  s.W = W;
  return s;
}

TileShape batch_shape_for(int precision, const BatchGridHost &g, int kind) {
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(std::make_tuple(precision, kind, batch_axis_len(g, kind)));
    if (it != g_tuned.end() && batch_shape_valid(precision, g, kind, it->second)) return it->second;
  }
  return batch_default_shape(precision, g, kind);
}

size_t batch_axis_bytes(int n, int precision) {
  const size_t csz = precision == FF_FP64 ? 16 : 8;
  auto r = [](size_t b) { return (b + 255) & ~size_t(255); };
  return r(n * csz) + (precision == FF_FP64 ? 0 : r(n * sizeof(double2))) + 2 * r(n * sizeof(int));
}

std::vector<int> batch_radix_order(int n, int order) {
  const std::vector<int> def = plan_factor_radices(n);
  std::vector<int> r = def;
  if (order == 1) {
    std::reverse(r.begin(), r.end());
  } else if (order == 2) {
    std::stable_partition(r.begin(), r.end(), [](int x) { return x == 5 || x == 3 || x == 7; });
  } else if (order != 0) {
    return {};
  }
  for (int q = 0; q < order; q++)
    if (batch_radix_order(n, q) == r) return {};
  return r;
}

int batch_axis_build(int n, int precision, int order, void *mem, AxisDev<double2> *ad, AxisDev<float2> *af,
                     cudaStream_t st) {
  const size_t csz = precision == FF_FP64 ? 16 : 8;
  auto r = [](size_t b) { return (b + 255) & ~size_t(255); };
  char *base = static_cast<char *>(mem);
  const size_t o_tw = 0;
  const size_t o_tw64 = precision == FF_FP64 ? o_tw : r(n * csz);
  const size_t o_rev = precision == FF_FP64 ? r(n * csz) : o_tw64 + r(n * sizeof(double2));
  const size_t o_ipos = o_rev + r(n * sizeof(int));
  const std::vector<int> radix = batch_radix_order(n, order);
  if (radix.empty()) return set_error(FF_ERR_INVALID, "radix order %d of length %d", order, n);
  const std::vector<int> rev = plan_digit_reversal(n, radix);
  std::vector<int> ipos(n);
  for (int q = 0; q < n; q++) ipos[rev[q]] = q;
  FF_CUDA(cudaMemcpyAsync(base + o_rev, rev.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
  FF_CUDA(cudaMemcpyAsync(base + o_ipos, ipos.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
  const int blocks = std::min(1024, (n + 255) / 256);
  k_twiddles<<<blocks, 256, 0, st>>>(n, reinterpret_cast<double2 *>(base + o_tw64));
  if (precision == FF_FP32) k_twiddles<<<blocks, 256, 0, st>>>(n, reinterpret_cast<float2 *>(base + o_tw));
  FF_CUDA(cudaGetLastError());
  // the host vectors above must outlive the copies
  FF_CUDA(cudaStreamSynchronize(st));
  *ad = AxisDev<double2>{};
  *af = AxisDev<float2>{};
  ad->n = af->n = n;
  ad->nstages = af->nstages = (int)radix.size();
  for (size_t q = 0; q < radix.size(); q++) ad->radix[q] = af->radix[q] = radix[q];
  ad->tw = reinterpret_cast<const double2 *>(base + o_tw);
  af->tw = reinterpret_cast<const float2 *>(base + o_tw);
  ad->tw64 = af->tw64 = reinterpret_cast<const double2 *>(base + o_tw64);
  ad->rev = af->rev = reinterpret_cast<const int *>(base + o_rev);
  ad->ipos = af->ipos = reinterpret_cast<const int *>(base + o_ipos);
  return FF_OK;
}

void batch_grid_init(BatchGridHost &h, const int n[3], const double *lo, const double *hi, int precision) {
  std::memset(&h, 0, sizeof(h));
  for (int d = 0; d < 3; d++) {
    h.n[d] = n[d];
    // ParisPencil.cpp:9-11; the reference domain [-pi, pi - 2pi/n] when no bounds are given
    const double len = (lo && hi) ? hi[d] - lo[d] : 2.0 * M_PI * double(n[d] - 1) / double(n[d]);
    h.dd[d] = n[d] > 1 ? 2.0 * M_PI * double(n[d] - 1) / (double(n[d]) * len) : 0.0;
  }
  h.nh = h.n[2] / 2 + 1;
  h.nhp = precision == FF_FP64 ? h.nh : (h.nh + 1) & ~1;
  h.invN = 1.0 / (double(h.n[0]) * double(h.n[1]) * double(h.n[2]));
  // TMA boxes: the largest divisor of the line length up to 256 rows
  for (int x = 0; x < 2; x++) {
    const int n = x == 0 ? h.n[1] : h.n[0];
    int d = std::min(n, 256);
    while (n % d) d--;
    h.box_rows[x] = d;
  }
}

int batch_grid_maps(const BatchGridHost &g, int precision, CUtensorMap maps[2]) {
  const size_t esz = precision == FF_FP64 ? 8 : 4;
  const int w1 = 128 / (int)(2 * esz);
  for (int x = 0; x < 2; x++) {
    const int rc = encode_spectrum_map(g.potential, g.n[0], g.n[1], g.nh, g.nhp, esz, w1, g.box_rows[x], x == 1,
                                       &maps[x]);
    if (rc != FF_OK) return rc;
  }
  return FF_OK;
}

size_t batch_grid_bytes(const BatchGridHost &h, int precision) {
  const size_t csz = precision == FF_FP64 ? 16 : 8;
  const size_t spec = (size_t)h.n[0] * h.n[1] * h.nhp * csz;
  const size_t real = (size_t)h.n[0] * h.n[1] * h.n[2] * (csz / 2);
  return std::max(spec, real);
}

int batch_check_dims(const int n[3], const double *lo, const double *hi, const char *who, int g) {
  for (int d = 0; d < 3; d++) {
    if (n[d] < 1) return set_error(FF_ERR_INVALID, "%s: grid %d n[%d] = %d < 1", who, g, d, n[d]);
    if (n[d] > FF_MAX_AXIS || !smooth2357(n[d]))
      return set_error(FF_ERR_UNSUPPORTED, "%s: grid %d n[%d] = %d is not 2^a 3^b 5^c 7^d <= %d", who, g, d,
                       n[d], FF_MAX_AXIS);
    if (lo && hi && n[d] > 1 && !(hi[d] > lo[d]))
      return set_error(FF_ERR_INVALID, "%s: grid %d hi[%d] <= lo[%d]", who, g, d, d);
    // the narrowest tile of a strided pass holds whole lines of 128-byte rows
    if ((size_t)n[d] * 128 + 128 > kBatchSmem)
      return set_error(FF_ERR_UNSUPPORTED, "%s: grid %d axis of %d points exceeds the batch tiles (%zu)", who, g,
                       n[d], (kBatchSmem - 128) / 128);
  }
  return FF_OK;
}

namespace {

// Work lists, block counts and shared memory of every pass from the grids'
// current shapes; uploads lists and descriptors (synchronously).
// Points every grid's axes at the tables of the radix order its owning pass
// uses (z: pass 0, y: pass 1, x: pass 2), building missing ones.
int apply_orders(ff_batch *b) {
  static const int owner[3] = {2, 1, 0};   // axis d is owned by pass owner[d]
  for (auto &g : b->grids) {
    for (int d = 0; d < 3; d++) {
      const int order = g.shape[owner[d]].order;
      auto key = std::make_pair(g.n[d], order);
      auto it = b->tables.find(key);
      if (it == b->tables.end()) {
        void *mem = nullptr;
        FF_CUDA(cudaMalloc(&mem, batch_axis_bytes(g.n[d], b->precision)));
        b->extra.push_back(mem);
        AxisDev<double2> ad;
        AxisDev<float2> af;
        const int rc = batch_axis_build(g.n[d], b->precision, order, mem, &ad, &af, b->cap);
        if (rc != FF_OK) return rc;
        it = b->tables.emplace(key, std::make_pair(ad, af)).first;
      }
      g.axd[d] = it->second.first;
      g.axf[d] = it->second.second;
    }
  }
  return FF_OK;
}

int build_work(ff_batch *b) {
  {
    const int rc = apply_orders(b);
    if (rc != FF_OK) return rc;
  }
  for (int k = 0; k < 5; k++) {
    std::vector<int> ent(b->count);
    std::vector<int> start(b->count + 1, 0);
    size_t smem = 256;
    for (int g = 0; g < b->count; g++) {
      ent[g] = g;
      start[g + 1] = start[g] + batch_tiles_of(b->grids[g], k);
      smem = std::max(smem, batch_shape_smem(b->precision, b->grids[g], k, b->grids[g].shape[k]));
    }
    b->ntiles[k] = start[b->count];
    b->smem[k] = smem;
    int per_sm = 0;
    int rc = pass_prepare(b->precision, k, smem, &per_sm);
    if (rc != FF_OK) return rc;
    if (per_sm < 1) return set_error(FF_ERR_UNSUPPORTED, "batch pass %d: a tile does not fit on an SM", k);
    b->ahead[k] = per_sm * b->num_sms;
    FF_CUDA(cudaMemcpy(b->entries[k], ent.data(), ent.size() * sizeof(int), cudaMemcpyHostToDevice));
    FF_CUDA(cudaMemcpy(b->starts[k], start.data(), start.size() * sizeof(int), cudaMemcpyHostToDevice));
  }
  b->desc_dirty = true;
  return FF_OK;
}

void drop_graph(ff_batch *b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
}

// The five passes (and the phase events), as
// issued on `st`; captured once into the graph.  The events are recorded as
// external event nodes, so the host can wait on and time them after a replay.
int issue_passes(ff_batch *b, cudaStream_t st) {
  FF_CUDA(cudaEventRecordWithFlags(b->ev[0], st, cudaEventRecordExternal));
  for (int k = 0; k < 5; k++) {
    int rc = pass_launch(b, k, st);
    if (rc != FF_OK) return rc;
    FF_CUDA(cudaEventRecordWithFlags(b->ev[k + 1], st, cudaEventRecordExternal));
  }
  return FF_OK;
}

int capture(ff_batch *b) {
  drop_graph(b);
  FF_CUDA(cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeThreadLocal));
  int rc = issue_passes(b, b->cap);
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamEndCapture(b->cap, &g);
  if (rc != FF_OK) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return set_error(FF_ERR_CUDA, "batch graph capture failed: %s", cudaGetErrorString(e));
  b->graph = g;
  FF_CUDA(cudaGraphInstantiate(&b->exec, g, 0));
  return FF_OK;
}

// Points the descriptors at the caller's buffers; marks them for upload if
// anything changed.
int set_buffers(ff_batch *b, void *const *density, void *const *potential) {
  for (int g = 0; g < b->count; g++) {
    if (!density[g] || !potential[g]) return set_error(FF_ERR_INVALID, "ff_batch: null buffer for grid %d", g);
    if (density[g] == potential[g]) return set_error(FF_ERR_INVALID, "ff_batch: grid %d density == potential", g);
    if (((uintptr_t)density[g] | (uintptr_t)potential[g]) & 15)
      return set_error(FF_ERR_INVALID, "ff_batch: grid %d buffers must be 16-byte aligned", g);
    if (b->grids[g].density != density[g] || b->grids[g].potential != potential[g]) {
      b->grids[g].density = density[g];
      b->grids[g].potential = potential[g];
      b->desc_dirty = true;
    }
  }
  return FF_OK;
}

int upload_desc(ff_batch *b, cudaStream_t st) {
  if (!b->desc_dirty) return FF_OK;
  for (int g = 0; g < b->count; g++) {
    desc_fill(b->precision, b->desc_host + g * b->desc_size, b->grids[g]);
    const int rc = batch_grid_maps(b->grids[g], b->precision, b->maps_host + 2 * g);
    if (rc != FF_OK) return rc;
  }
  FF_CUDA(cudaMemcpyAsync(b->desc, b->desc_host, b->count * b->desc_size, cudaMemcpyHostToDevice, st));
  FF_CUDA(cudaMemcpyAsync(b->maps, b->maps_host, 2 * b->count * sizeof(CUtensorMap), cudaMemcpyHostToDevice, st));
  // the pinned image may be rewritten by the next call only after this copy
  FF_CUDA(cudaStreamSynchronize(st));
  b->desc_dirty = false;
  return FF_OK;
}

int take_status(ff_batch *b, cudaStream_t st) {
  int h = 0;
  FF_CUDA(cudaMemcpyAsync(&h, b->status, sizeof(int), cudaMemcpyDeviceToHost, st));
  FF_CUDA(cudaStreamSynchronize(st));
  if (h != kDevOk) {
    FF_CUDA(cudaMemsetAsync(b->status, 0, sizeof(int), st));
    FF_CUDA(cudaStreamSynchronize(st));
    return set_error(FF_ERR_TIMEOUT, "a batch tile's bulk copy did not complete within its wait limit");
  }
  return FF_OK;
}

// Median of `reps` timed launches of pass `kind` (after one warm-up).
int time_pass(ff_batch *b, int kind, cudaStream_t st, int reps, float *ms) {
  std::vector<float> t;
  for (int r = 0; r <= reps; r++) {
    FF_CUDA(cudaEventRecord(b->ev[0], st));
    int rc = pass_launch(b, kind, st);
    if (rc != FF_OK) return rc;
    FF_CUDA(cudaEventRecord(b->ev[1], st));
    FF_CUDA(cudaEventSynchronize(b->ev[1]));
    float x = 0;
    FF_CUDA(cudaEventElapsedTime(&x, b->ev[0], b->ev[1]));
    if (r > 0) t.push_back(x);
  }
  std::sort(t.begin(), t.end());
  *ms = t[t.size() / 2];
  return FF_OK;
}


// The batched grids' tables, descriptors, work lists and events (count >= 1
// grids that batch_check_dims accepted).  On failure the caller destroys b.
int batch_create_core(ff_batch *b, int count, const int *dims, const double *lo, const double *hi,
                      int precision) {
  b->count = count;
  b->desc_size = desc_size(precision);
  // distinct axis lengths -> one table set each
  std::map<int, size_t> table_of;
  size_t off = 0;
  auto take = [&](size_t bytes) { size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
  for (int g = 0; g < count; g++)
    for (int d = 0; d < 3; d++) {
      const int n = dims[3 * g + d];
      if (!table_of.count(n)) table_of[n] = take(batch_axis_bytes(n, precision));
    }
  const size_t o_status = take(sizeof(int));
  const size_t o_desc = take((size_t)count * b->desc_size);
  const size_t o_maps = take((size_t)count * 2 * sizeof(CUtensorMap));
  size_t o_ent[5], o_start[5];
  for (int k = 0; k < 5; k++) {
    o_ent[k] = take((size_t)count * sizeof(int));
    o_start[k] = take((size_t)(count + 1) * sizeof(int));
  }
  b->dmem_size = off;
  if (cudaMalloc(&b->dmem, off) != cudaSuccess) {
    cudaGetLastError();
    b->dmem = nullptr;
    return set_error(FF_ERR_NOMEM, "ff_batch_create: cudaMalloc(%zu) for tables failed", off);
  }
  if (cudaMallocHost((void **)&b->desc_host, (size_t)count * b->desc_size) != cudaSuccess ||
      cudaMallocHost((void **)&b->maps_host, (size_t)count * 2 * sizeof(CUtensorMap)) != cudaSuccess) {
    cudaGetLastError();
    return set_error(FF_ERR_NOMEM, "ff_batch_create: pinned descriptor image");
  }
  char *base = static_cast<char *>(b->dmem);
  b->status = reinterpret_cast<int *>(base + o_status);
  b->desc = base + o_desc;
  b->maps = reinterpret_cast<CUtensorMap *>(base + o_maps);
  for (int k = 0; k < 5; k++) {
    b->entries[k] = reinterpret_cast<int *>(base + o_ent[k]);
    b->starts[k] = reinterpret_cast<int *>(base + o_start[k]);
  }
  int rc = FF_OK;
  if (cudaMemset(b->status, 0, sizeof(int)) != cudaSuccess) rc = set_error(FF_ERR_CUDA, "ff_batch_create: memset");
  if (rc == FF_OK && cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking) != cudaSuccess)
    rc = set_error(FF_ERR_CUDA, "ff_batch_create: stream");
  // axis tables: twiddles from FP64 sincospi, digit reversal of the default plan
  std::map<int, std::pair<AxisDev<double2>, AxisDev<float2>>> axes;
  for (const auto &t : table_of) {
    if (rc != FF_OK) break;
    AxisDev<double2> ad;
    AxisDev<float2> af;
    rc = batch_axis_build(t.first, precision, 0, base + t.second, &ad, &af, b->cap);
    axes[t.first] = std::make_pair(ad, af);
    b->tables[std::make_pair(t.first, 0)] = std::make_pair(ad, af);
  }
  b->grids.resize(count);
  b->bytes.resize(count);
  for (int g = 0; g < count && rc == FF_OK; g++) {
    BatchGridHost &h = b->grids[g];
    batch_grid_init(h, dims + 3 * g, lo ? lo + 3 * g : nullptr, hi ? hi + 3 * g : nullptr, precision);
    for (int d = 0; d < 3; d++) {
      h.axd[d] = axes[h.n[d]].first;
      h.axf[d] = axes[h.n[d]].second;
    }
    h.status = b->status;
    b->bytes[g] = batch_grid_bytes(h, precision);
    for (int k = 0; k < 5; k++) h.shape[k] = batch_shape_for(precision, h, k);
  }
  if (rc == FF_OK) rc = build_work(b);
  return rc;
}

// A grid the batch kernels take: every axis 2^a 3^b 5^c 7^d and short enough
// for their tiles (batch_check_dims).
bool batchable(const int n[3]) {
  for (int d = 0; d < 3; d++)
    if (!smooth2357(n[d]) || (size_t)n[d] * 128 + 128 > kBatchSmem) return false;
  return true;
}

}  // namespace
}  // namespace ff

extern "C" {

int ff_batch_create(int count, const int *dims, const double *lo, const double *hi, int precision, ff_batch **out) {
  if (!out) return set_error(FF_ERR_INVALID, "ff_batch_create: null output");
  *out = nullptr;
  if (count < 1 || !dims) return set_error(FF_ERR_INVALID, "ff_batch_create: count %d or dims missing", count);
  if (precision != FF_FP64 && precision != FF_FP32)
    return set_error(FF_ERR_INVALID, "ff_batch_create: precision %d is neither FF_FP64 nor FF_FP32", precision);
  std::vector<int> bdims;
  std::vector<double> blo, bhi;
  for (int g = 0; g < count; g++) {
    const int *n = dims + 3 * g;
    for (int d = 0; d < 3; d++) {
      if (n[d] < 1) return set_error(FF_ERR_INVALID, "ff_batch_create: grid %d n[%d] = %d < 1", g, d, n[d]);
      if (n[d] > FF_MAX_AXIS)
        return set_error(FF_ERR_UNSUPPORTED, "ff_batch_create: grid %d n[%d] = %d is above %d", g, d, n[d],
                         FF_MAX_AXIS);
      if (lo && hi && n[d] > 1 && !(hi[3 * g + d] > lo[3 * g + d]))
        return set_error(FF_ERR_INVALID, "ff_batch_create: grid %d hi[%d] <= lo[%d]", g, d, d);
    }
  }
  ff_batch *b = new ff_batch();
  b->user_count = count;
  b->precision = precision;
  b->csz = precision == FF_FP64 ? 16 : 8;
  if (cudaGetDevice(&b->device) != cudaSuccess ||
      cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, b->device) != cudaSuccess) {
    delete b;
    return set_error(FF_ERR_CUDA, "ff_batch_create: no current CUDA device");
  }
  int rc = FF_OK;
  b->where.resize(count);
  for (int g = 0; g < count && rc == FF_OK; g++) {
    const int *n = dims + 3 * g;
    if (batchable(n)) {
      b->where[g] = (int)(bdims.size() / 3);
      for (int d = 0; d < 3; d++) {
        bdims.push_back(n[d]);
        if (lo && hi) {
          blo.push_back(lo[3 * g + d]);
          bhi.push_back(hi[3 * g + d]);
        }
      }
    } else {
      // the reference domain of the grid unless bounds are given
      double glo[3], ghi[3];
      for (int d = 0; d < 3; d++) {
        glo[d] = lo && hi ? lo[3 * g + d] : -M_PI;
        ghi[d] = lo && hi ? hi[3 * g + d] : M_PI - 2.0 * M_PI / n[d];
      }
      ff_plan *pl = nullptr;
      rc = ff_plan_create(n, glo, ghi, precision, &pl);
      if (rc != FF_OK) break;
      size_t nb = 0;
      ff_plan_bytes(pl, &nb);
      b->where[g] = -(int)b->side.size() - 1;
      b->side.push_back(pl);
      b->side_bytes.push_back(nb);
    }
  }
  const int nb = (int)(bdims.size() / 3);
  if (rc == FF_OK && nb > 0)
    rc = batch_create_core(b, nb, bdims.data(), lo && hi ? blo.data() : nullptr, lo && hi ? bhi.data() : nullptr,
                           precision);
  for (int e = 0; e < 6 && rc == FF_OK; e++)
    if (cudaEventCreate(&b->ev[e]) != cudaSuccess) rc = set_error(FF_ERR_CUDA, "ff_batch_create: event");
  for (int e = 0; e < 2 && rc == FF_OK; e++)
    if (cudaEventCreate(&b->side_ev[e]) != cudaSuccess) rc = set_error(FF_ERR_CUDA, "ff_batch_create: event");
  if (rc != FF_OK) {
    ff_batch_destroy(b);
    return rc;
  }
  *out = b;
  return FF_OK;
}

int ff_batch_bytes(const ff_batch *b, int index, size_t *bytes) {
  if (!b || !bytes) return set_error(FF_ERR_INVALID, "ff_batch_bytes: null argument");
  if (index < 0 || index >= b->user_count) return set_error(FF_ERR_INVALID, "ff_batch_bytes: index %d", index);
  const int w = b->where[index];
  *bytes = w >= 0 ? b->bytes[w] : b->side_bytes[-w - 1];
  return FF_OK;
}

int ff_batch_shape(const ff_batch *b, int index, int kind, int *W, int *ct, int *tma) {
  if (!b || index < 0 || index >= b->user_count || kind < 0 || kind > 4)
    return set_error(FF_ERR_INVALID, "ff_batch_shape: bad argument");
  const int w = b->where[index];
  if (w < 0)
    return set_error(FF_ERR_UNSUPPORTED, "ff_batch_shape: grid %d runs through its own single-grid plan", index);
  if (W) *W = b->grids[w].shape[kind].W;
  if (ct) *ct = b->grids[w].shape[kind].ct;
  if (tma) *tma = b->grids[w].shape[kind].tma;
  return FF_OK;
}

int ff_batch_radices(const ff_batch *b, int index, int axis, int radix[16], int *count) {
  if (!b || index < 0 || index >= b->user_count || axis < 0 || axis > 2 || !radix || !count)
    return set_error(FF_ERR_INVALID, "ff_batch_radices: bad argument");
  if (b->where[index] < 0)
    return set_error(FF_ERR_UNSUPPORTED, "ff_batch_radices: grid %d runs through its own single-grid plan", index);
  const AxisDev<double2> &ax = b->grids[b->where[index]].axd[axis];
  *count = ax.nstages;
  for (int q = 0; q < ax.nstages; q++) radix[q] = ax.radix[q];
  return FF_OK;
}

}  // extern "C"

namespace ff {
namespace {

// The caller's per-grid buffers split into the batched grids' arrays.
int split_buffers(const ff_batch *b, void *const *density, void *const *potential, std::vector<void *> &bd,
                  std::vector<void *> &bp) {
  bd.assign(b->count, nullptr);
  bp.assign(b->count, nullptr);
  for (int u = 0; u < b->user_count; u++) {
    if (!density[u] || !potential[u]) return set_error(FF_ERR_INVALID, "ff_batch: null buffer for grid %d", u);
    if (b->where[u] >= 0) {
      bd[b->where[u]] = density[u];
      bp[b->where[u]] = potential[u];
    }
  }
  return FF_OK;
}

int batch_status(ff_batch *b, cudaStream_t st) {
  int rc = b->count > 0 ? take_status(b, st) : FF_OK;
  for (ff_plan *pl : b->side) {
    const int r2 = ff_plan_check(pl, st);
    if (rc == FF_OK) rc = r2;
  }
  return rc;
}

}  // namespace
}  // namespace ff

extern "C" {

int ff_batch_solve(ff_batch *b, void *const *density, void *const *potential, void *stream, ff_phase_times *times) {
  if (!b || !density || !potential) return set_error(FF_ERR_INVALID, "ff_batch_solve: null argument");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<void *> bd, bp;
  int rc = split_buffers(b, density, potential, bd, bp);
  if (rc != FF_OK) return rc;
  if (b->count > 0) {
    rc = set_buffers(b, bd.data(), bp.data());
    if (rc == FF_OK) rc = upload_desc(b, st);
    if (rc == FF_OK && !b->exec) rc = capture(b);
    if (rc != FF_OK) return rc;
  }
  if (times && b->count == 0) FF_CUDA(cudaEventRecord(b->side_ev[0], st));
  if (b->count > 0) FF_CUDA(cudaGraphLaunch(b->exec, st));
  for (int u = 0; u < b->user_count; u++) {
    const int w = b->where[u];
    if (w >= 0) continue;
    rc = ff_solve(b->side[-w - 1], b->side_bytes[-w - 1], density[u], potential[u], stream, nullptr);
    if (rc != FF_OK) return rc;
  }
  if (times) {
    FF_CUDA(cudaEventRecord(b->side_ev[1], st));
    FF_CUDA(cudaEventSynchronize(b->side_ev[1]));
    // per pass: the batched grids' five launches (zero if none); total: the
    // whole solve, single-grid plans of the other grids included
    times->count = 5;
    for (int k = 0; k < 5; k++) {
      float ms = 0;
      if (b->count > 0) FF_CUDA(cudaEventElapsedTime(&ms, b->ev[k], b->ev[k + 1]));
      times->ms[k] = ms;
    }
    float tot = 0;
    FF_CUDA(cudaEventElapsedTime(&tot, b->count > 0 ? b->ev[0] : b->side_ev[0], b->side_ev[1]));
    times->total_ms = tot;
    return batch_status(b, st);
  }
  return FF_OK;
}

int ff_batch_check(ff_batch *b, void *stream) {
  if (!b) return set_error(FF_ERR_INVALID, "ff_batch_check: null batch");
  return batch_status(b, static_cast<cudaStream_t>(stream));
}

// Coordinate search over tile shapes: for each pass and each axis length
// used by that pass, every valid candidate shape is applied to all grids of
// that length and the whole pass is timed; the fastest is kept (and
// remembered for later batches of this process).  Candidates: z passes
// W in {d/2, d, 2d} around the default d line pairs, strided passes 1, 2 or
// 4 rows of 128 bytes per tile row; each with the compile-time tile (where
// the length has one) and with the runtime plan.
int ff_batch_tune(ff_batch *b, void *const *density_u, void *const *potential_u, void *stream, int reps) {
  if (!b || !density_u || !potential_u) return set_error(FF_ERR_INVALID, "ff_batch_tune: null argument");
  if (reps < 1) reps = 3;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  std::vector<void *> bd, bp;   // the batched grids' buffers (grids with own plans are not tuned)
  int rc = split_buffers(b, density_u, potential_u, bd, bp);
  if (rc != FF_OK || b->count == 0) return rc;
  void *const *density = bd.data();
  void *const *potential = bp.data();
  rc = set_buffers(b, density, potential);
  if (rc != FF_OK) return rc;
  for (int g = 0; g < b->count; g++) {
    FF_CUDA(cudaMemsetAsync(density[g], 0, b->bytes[g], st));
    FF_CUDA(cudaMemsetAsync(potential[g], 0, b->bytes[g], st));
  }
  drop_graph(b);
  for (int k = 0; k < 5; k++) {
    std::vector<int> lens;
    for (const auto &g : b->grids) lens.push_back(batch_axis_len(g, k));
    std::sort(lens.begin(), lens.end());
    lens.erase(std::unique(lens.begin(), lens.end()), lens.end());
    for (int n : lens) {
      int first = -1;
      for (int g = 0; g < b->count; g++)
        if (batch_axis_len(b->grids[g], k) == n) { first = g; break; }
      const BatchGridHost &ref = b->grids[first];
      std::vector<TileShape> cand;
      const TileShape d = batch_default_shape(b->precision, ref, k);
      for (int ct = batch_special_n(n) ? 1 : 0; ct >= 0; ct--) {
        if (k == 0 || k == 4) {
          for (int W : {std::max(1, d.W / 2), d.W, d.W * 2}) {
            cand.push_back(TileShape{W, ct, 0, 0});
            if (!ct) cand.push_back(TileShape{W, 0, 1, 0});
          }
        } else {
          const int w1 = 128 / (int)b->csz;
          for (int m : {1, 2, 4}) cand.push_back(TileShape{m * w1, ct, 0, 0});
          cand.push_back(TileShape{w1, ct, 1, 0});
        }
      }
      // runtime plans of the pass that owns the axis: every radix order too
      if (k <= 2) {
        const size_t base_count = cand.size();
        for (int order = 1; order < kBatchOrders; order++) {
          if (batch_radix_order(n, order).empty()) continue;
          for (size_t q = 0; q < base_count; q++)
            if (!cand[q].ct) {
              TileShape c = cand[q];
              c.order = order;
              cand.push_back(c);
            }
        }
      }
      // the shape in use is timed first and kept unless a candidate beats it
      // by more than 3 % (passes of near-equal candidates differ by noise)
      TileShape best = ref.shape[k];
      float best_ms = 1e30f;
      cand.insert(cand.begin(), best);
      for (size_t ci = 0; ci < cand.size(); ci++) {
        const TileShape &c = cand[ci];
        bool ok = true;
        for (const auto &g : b->grids)
          if (batch_axis_len(g, k) == n && !batch_shape_valid(b->precision, g, k, c)) ok = false;
        if (!ok) continue;
        for (auto &g : b->grids)
          if (batch_axis_len(g, k) == n) g.shape[k] = c;
        rc = build_work(b);
        if (rc == FF_OK) rc = upload_desc(b, st);
        float ms = 0;
        if (rc == FF_OK) rc = time_pass(b, k, st, reps, &ms);
        if (rc != FF_OK) return rc;
        if (ci == 0 || ms < 0.97f * best_ms) {
          best_ms = ms;
          best = c;
        }
      }
      for (auto &g : b->grids)
        if (batch_axis_len(g, k) == n) g.shape[k] = best;
      std::lock_guard<std::mutex> lk(g_tune_mu);
      g_tuned[std::make_tuple(b->precision, k, n)] = best;
    }
  }
  rc = build_work(b);
  if (rc == FF_OK) rc = upload_desc(b, st);
  if (rc == FF_OK) rc = take_status(b, st);
  return rc;
}

int ff_batch_destroy(ff_batch *b) {
  if (!b) return FF_OK;
  drop_graph(b);
  for (ff_plan *pl : b->side) ff_plan_destroy(pl);
  for (int e = 0; e < 2; e++)
    if (b->side_ev[e]) cudaEventDestroy(b->side_ev[e]);
  for (int e = 0; e < 6; e++)
    if (b->ev[e]) cudaEventDestroy(b->ev[e]);
  if (b->cap) cudaStreamDestroy(b->cap);
  if (b->desc_host) cudaFreeHost(b->desc_host);
  if (b->maps_host) cudaFreeHost(b->maps_host);
  int rc = FF_OK;
  for (void *m : b->extra) cudaFree(m);
  if (b->dmem && cudaFree(b->dmem) != cudaSuccess) rc = set_error(FF_ERR_CUDA, "ff_batch_destroy: cudaFree failed");
  delete b;
  return rc;
}

}  // extern "C"
