// Instantiates the real row kernels with compile-time radix sequences (float).
#include "rrows.cuh"

namespace ffb {
namespace rrows {
template cudaError_t launch<float>(const TileArgs<float> &, IoKind, cudaStream_t);
}  // namespace rrows
}  // namespace ffb
