// Instantiates the real row kernels with compile-time radix sequences (float).
#include "rrows.cuh"

namespace ffb {
namespace rrows {
template cudaError_t launch<float>(const TileArgs<float> &, IoKind, cudaStream_t);
template bool shape<float>(const TileArgs<float> &, IoKind, TileKernel *);
}  // namespace rrows
}  // namespace ffb
