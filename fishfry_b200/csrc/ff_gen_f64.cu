// FP64 kernels of the passes along axes without a compile-time plan.
#include "ff_gen_dev.cuh"

namespace ff {
FF_INSTANTIATE_GEN(double)
}  // namespace ff
