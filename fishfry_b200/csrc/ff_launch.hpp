// Launches of the solve's passes.
#pragma once

#include <cuda_runtime.h>

namespace ff {

// Launches k after the work queued on st, as a programmatic dependent of the
// kernel before it: once that kernel's blocks have all started (pdl_start), k's
// blocks take the places that its last ones free, set themselves up and wait in
// pdl_wait until it has completed and its writes are visible.  A pass's first
// blocks then need no launch after the last block of the pass before.  Every
// kernel launched this way calls pdl_wait on every thread before it touches
// memory that another launch reads or writes, so that its own completion implies
// that of all passes before it.
//
// Pass 1 depends in the same way on the caller's kernel before it (a plain launch
// there costs 2 us of a 57 us solve).  Its pdl_wait covers what was queued before
// that kernel too: a kernel that may start before its predecessor has completed
// has to wait for it (griddepcontrol.wait, PTX), so its completion implies the
// predecessor's.  The last kernel of every call does not call pdl_start: what a
// caller launches next starts after the call's work, however it is launched.
//
// chained = false is a plain launch, which a solve takes above kChainBytes of
// spectrum.  On one B200, plain / chained solves with the copy of their field:
// 64^3 FP64 29.1 / 20.6 us, FP32 26.5 / 20.5; 128^3 62.9 / 53.9, 49.2 / 41.0;
// 256^3 343 / 334, 209 / 199; 384^3 (455 MB FP64) 1226 / 1221, 686 / 679; from
// there on within the noise (480x400x360 1573 / 1575, 863 / 877; 512^3 2546 / 2546,
// 1423 / 1407; 1024x512x512 5393 / 5435, 2915 / 2901).
constexpr size_t kChainBytes = size_t(256) << 20;

template <typename... P, typename... A>
cudaError_t launch_chained(bool chained, void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                           A &&...a) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr;
  c.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&c, k, static_cast<P>(a)...);
}

}  // namespace ff
