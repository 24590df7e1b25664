// Instantiates the mixed-radix tile kernels (float, plain transforms).
#include "mixed.cuh"

namespace ffb {
namespace mixed {
template cudaError_t launch<float, 0>(const TileArgs<float> &, IoKind, size_t, cudaStream_t);
}  // namespace mixed
}  // namespace ffb
