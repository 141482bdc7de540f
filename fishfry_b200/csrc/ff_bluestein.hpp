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
  const C *chirp;    // chirp[j] = exp(-i*pi*j^2/n), j < n (FP64-generated)
  const C *ghat;     // ghat[pos] = G[k]/M for the frequency k at DIF output position pos,
                     // G the M-point DFT of g[m] = conj chirp[|m|] (|m| < n, indices mod M)
};

// The transform length M of an axis of n points.
int bs_padded_length(int n);

// Launch shape of pass `kind` (0 z forward, 1 y forward, 2 x, 3 y inverse,
// 4 z inverse) of an ni x nj x nk grid whose axis for that pass goes through
// M points.
GenShape bs_shape(int kind, int ni, int nj, int nk, int nhp, int esz, int M, int num_sms);

// Raises the pass kernel's shared-memory limit; FF_ERR_UNSUPPORTED if the tile
// does not fit.
template <typename T> int bs_prepare(int kind, size_t smem);

// Device tables of one axis: chirp (n values) and ghat (M values, from the
// M-point plan's group bases k0 and last radix).  Enqueued on the current
// device's default stream.
template <typename C> int bs_tables(int n, int M, const int *k0, int last_radix, C *chirp, C *ghat);

// Pass launches.  in and out are the pass's arrays as the regular passes use
// them: z forward reads the real field and writes the spectrum; y forward and
// x work in place on the spectrum; y inverse reads one spectrum array and
// writes the other; z inverse reads the spectrum and writes the real field.
template <typename T>
int bs_launch(int kind, const BsPass<typename Cplx<T>::type> &a, const GenShape &s, const void *in, void *out,
              cudaStream_t st);

}  // namespace ff
