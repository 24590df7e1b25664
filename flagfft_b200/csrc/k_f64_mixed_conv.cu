// Instantiates the mixed-radix tile kernels (double, convolutions).
#include "mixed.cuh"

namespace ffb {
namespace mixed {
template cudaError_t launch<double, 1>(const TileArgs<double> &, IoKind, size_t, cudaStream_t);
template cudaError_t launch<double, 2>(const TileArgs<double> &, IoKind, size_t, cudaStream_t);
template cudaError_t launch<double, 3>(const TileArgs<double> &, IoKind, size_t, cudaStream_t);
}  // namespace mixed
}  // namespace ffb
