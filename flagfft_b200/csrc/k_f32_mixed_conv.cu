// Instantiates the mixed-radix tile kernels (float, convolutions).
#include "mixed.cuh"

namespace ffb {
namespace mixed {
template cudaError_t launch<float, 1>(const TileArgs<float> &, IoKind, size_t, cudaStream_t);
template cudaError_t launch<float, 2>(const TileArgs<float> &, IoKind, size_t, cudaStream_t);
template cudaError_t launch<float, 3>(const TileArgs<float> &, IoKind, size_t, cudaStream_t);
}  // namespace mixed
}  // namespace ffb
