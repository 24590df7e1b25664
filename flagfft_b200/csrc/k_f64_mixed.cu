// Instantiates the mixed-radix tile kernels (double, plain transforms).
#include "mixed.cuh"

namespace ffb {
namespace mixed {
template cudaError_t launch<double, 0>(const TileArgs<double> &, IoKind, size_t, cudaStream_t);
}  // namespace mixed
}  // namespace ffb
