// Passes along axes without a compile-time plan (2^a 3^b 5^c 7^d lengths other
// than the specialised ones): plans and launch shapes, shared by the host code
// (ff_gen.cu) and the kernels (ff_gen_dev.cuh).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <vector>

#include "ff_fft.cuh"

namespace ff {

constexpr int kGenMaxStages = 8;   // 7-smooth lengths up to 4096: at most 5 with the radices below
constexpr int kGenMaxRadix = 10;
constexpr int kGenSplitRadix = 7;  // last stage of the z passes: two groups per thread

// One stage of a plan as the kernels walk it (DIF order: stage 0 spans the
// line).  The items of a column are its n/R butterflies; a thread takes items
// b0, b0 + step, ... and keeps (b / m, b % m) by adding (dq, dr).
struct GenStage {
  int R;        // radix
  int L, m;     // span and m = L / R, the distance between a butterfly's points
  int nb;       // butterflies per column, n / R
  int dq, dr;   // step / m, step % m
  float inv_m;  // 1 / m, correctly rounded
  float inv_nb; // tiles with butterflies fastest (gen_line_stages): 1 / nb
  int ms;       // rows of the tile between a butterfly's points
  float inv_pb; // z passes: 1 / blocks of this stage in a block of stage 0 (0: rows are not padded)
  int tw;       // offset of the stage's twiddles in the table (complex values)
};

// One axis as the kernels see it.  Twiddles are stored per stage as
// [j][r], r < Rp = R rounded up to even: entry (j, r) = exp(-2 pi i j r / L).
template <typename C> struct GenAxis {
  int n, S;
  GenStage st[kGenMaxStages + 1];   // gen_line_stages: st[S] counts the split's items
  const C *tw;        // per-stage twiddles, in C's precision (FP64-generated)
  // strided passes: last-stage group g -> frequency base k0 (the group's R
  // frequencies are k0 + r n/R); z passes: k0 -> first tile row of its group
  const int *idx;
};

// Rows between the blocks of stage 0 in a z tile beyond their length: 1 where
// that makes their distance odd.  The groups of consecutive frequency bases,
// which a warp of the last stage reads together, lie one such distance apart
// (digit reversal); an even one put them in the same banks (a 40 % share of
// conflicted wavefronts at 480x400x360).
int gen_pad(int n, const std::vector<int> &radix);

// Radix split of a 2^a 3^b 5^c 7^d length in DIF order.  split: the last radix
// is at most kGenSplitRadix.
std::vector<int> gen_radices(int n, bool split);

// Frequency base of each group of the last stage.
std::vector<int> gen_bases(int n, const std::vector<int> &radix);

// Complex values of the twiddle table, and the stage descriptors for blocks of
// `threads` threads on tiles of `units` columns (threads a multiple of units);
// pad: gen_pad for z tiles, 0 for strided ones.
int gen_table_size(int n, const std::vector<int> &radix);
void gen_stages(int n, const std::vector<int> &radix, int pad, int threads, int units, int *S, GenStage *st);

// The same for z tiles with butterflies fastest (ff_gen_lines.cuh): a thread
// takes items t, t + threads, ... of all columns and keeps (column, butterfly) by
// adding (dq, dr) = (threads / nb, threads % nb); st[S] counts the items of the
// forward split.  table: the twiddle steps of an axis's plain table instead of
// packed offsets.  Shared memory of such a tile of W line pairs.
void gen_line_stages(int n, const std::vector<int> &radix, int pad, int threads, bool table, int *S, GenStage *st);
size_t gen_line_smem(int nk, int nhp, int esz, int tile_rows, int W);

// A tile is `units` columns of 16 bytes (one FP64 or two adjacent FP32 complex
// values; z passes: one FP64 line pair or two FP32 ones) by n rows.
struct GenShape {
  int units;      // 1, 2, 4 or 8
  int threads;
  size_t smem;
  long grid;
  bool chained;   // launched as a programmatic dependent (ff_launch.hpp)
  int box_rows;   // strided passes: rows per TMA box
  int tile_rows;  // z passes
  int lp, sp;     // z passes: pitch of a staged real line (values), of a staged spectrum row (complex values)
};

// Launch shape of pass `kind` (0 z fwd, 1 y fwd, 2 x, 3 y inv, 4 z inv) of an
// ni x nj x nk grid; esz: bytes of a real value.
GenShape gen_shape(int kind, int ni, int nj, int nk, int nhp, int esz, const std::vector<int> &radix, int num_sms);

// Parts of gen_shape that other tiles share: units, pitches, shared memory and
// grid of a z pass whose tile has s->tile_rows rows (lines_kind: a tile with
// butterflies fastest), the most units that keep `limit` bytes of shared memory;
// threads per block from the shared memory.
void gen_z_shape(GenShape *s, int ni, int nj, int nk, int nhp, int esz, int num_sms, bool lines_kind, size_t limit);
void gen_pick_threads(GenShape *s);

// Cost of an n-point transform's stages per point (arbitrary unit).
double gen_cost(int n);

// What the pass kernels need besides the axis.
template <typename C> struct GenPass {
  int ni, nj, nk, nh, nhp;
  int lu;              // log2 of the tile's units
  int box_rows;
  int tile_rows;       // z passes: padded rows
  int lp, sp;
  int per_line;        // z passes: real lines move by one bulk copy each (16-byte multiples), else as one block
  double dd[3], invN;
  int *status;
  int wait_iters;
  int l2_ahead;        // z passes: blocks ahead whose input is hinted into L2
  GenAxis<C> ax;
};

// The index table of an axis (GenAxis::idx), host side, n / (last radix) values.
void gen_index(int n, const std::vector<int> &radix, int pad, bool by_frequency, std::vector<int> *out);

// Fills the twiddle table of one axis at `mem` (gen_axis_bytes) on the default
// stream and points ax at it and at the device copy of its index table.
size_t gen_axis_bytes(int n, const std::vector<int> &radix, int esz);
template <typename C> int gen_axis_build(int n, const std::vector<int> &radix, void *mem, const int *idx, GenAxis<C> *ax);

// Raises the pass kernel's shared-memory limit; FF_ERR_UNSUPPORTED if it does
// not fit.
template <typename T> int gen_prepare(int kind, size_t smem);

// Launches pass `kind`: z fwd reads `in` (real) and writes `out` (spectrum),
// z inv the reverse; the strided passes read the spectrum of `map` and write
// `out` (y) or the same spectrum (x).
template <typename T>
int gen_launch(int kind, const GenPass<typename Cplx<T>::type> &a, const GenShape &s, const CUtensorMap *map,
               const void *in, void *out, cudaStream_t st);

}  // namespace ff
