// Axes whose length has a prime factor above 7 (single-grid solve).
//
// cuFFT, which the reference calls for every line transform
// (ParisPencil.cpp:78-81 plans, :165/:212/:259/:288/:334/:380 executions),
// accepts any length.  Here an axis of n points with a prime factor above 7
// is transformed by Bluestein's algorithm: with the chirp
// c[j] = exp(-i*pi*j^2/n), the forward DFT is
//   X[k] = c[k] * sum_j (x[j] c[j]) conj c[k-j],
// a circular convolution of M >= 2n-1 points (M = 2^a 3^b 5^c 7^d), computed by
// the stages of the generic passes (ff_gen_stages.cuh): an M-point forward DIF
// transform of the premultiplied, zero-padded line, a product with the
// transform of the convolution kernel (one register group, with the last DIF
// and first DIT stages), an M-point inverse DIT transform, and the
// postmultiplication.  The inverse DFT uses the conjugate chirp and kernel.
// A prime n whose n - 1 has only the factors 2, 3, 5 and 7 goes through Rader's
// algorithm instead: with a primitive root g of n and w = exp(-2*pi*i/n),
//   X[g^-s] = x[0] + sum_q x[g^q] w^(g^-(s-q)),  X[0] = x[0] + sum_q x[g^q],
// a circular convolution of n - 1 points: half the points of Bluestein's and
// no chirp.  The inverse DFT takes X in that order, and the conjugate kernel.
// Each pass keeps its own work around the transform: the z pass packs two
// real lines into one complex line and splits the result into the two half
// spectra (and the reverse), the x pass applies the filter between its
// forward and inverse transforms.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "ff_gen.hpp"

namespace ff {

// Pass arguments: those of the generic passes, whose axis is the M-point
// transform, and
template <typename C> struct BsPass : GenPass<C> {
  int n;             // axis length
  const int *perm;   // Rader: perm[q] = g^q mod n, q < n - 1 (null: Bluestein)
  const C *chirp;    // chirp[j] = exp(-i*pi*j^2/n), j < n (FP64-generated)
  const C *ghat;     // ghat[pos] = G[k]/M for the frequency k at DIF output position pos,
                     // G the M-point DFT of g[m] = conj chirp[|m|] (|m| < n, indices mod M);
                     // Rader: of w^(g^-m), w = exp(-2*pi*i/n)
};

// The smallest primitive root of n where Rader's algorithm applies, else 0.
int rader_root(int n);

// The transform length M of an axis of n points by Bluestein's algorithm.
int bs_padded_length(int n);

// Launch shape of pass `kind` (0 z forward, 1 y forward, 2 x, 3 y inverse,
// 4 z inverse) of an ni x nj x nk grid whose axis for that pass takes tiles of
// `rows` points (M, or n for Rader: its n - 1 points and point 0).
GenShape bs_shape(int kind, int ni, int nj, int nk, int nhp, int esz, int rows, int num_sms);

// Raises the pass kernel's shared-memory limit; FF_ERR_UNSUPPORTED if the tile
// does not fit.
template <typename T> int bs_prepare(int kind, bool rader, size_t smem);

// Device tables of one axis: chirp (n values) and ghat (M values, from the
// M-point plan's group bases k0 and last radix).  Enqueued on the current
// device's default stream.
template <typename C> int bs_tables(int n, int M, const int *k0, int last_radix, C *chirp, C *ghat);
// The same for Rader: ghat (n - 1 values) from perm and the (n-1)-point plan.
template <typename C> int rader_tables(int n, const int *perm, const int *k0, int last_radix, C *ghat);

// Pass launches.  in and out are the pass's arrays as the regular passes use
// them: z forward reads the real field and writes the spectrum; y forward and
// x work in place on the spectrum; y inverse reads one spectrum array and
// writes the other; z inverse reads the spectrum and writes the real field.
template <typename T>
int bs_launch(int kind, const BsPass<typename Cplx<T>::type> &a, const GenShape &s, const void *in, void *out,
              cudaStream_t st);

}  // namespace ff
