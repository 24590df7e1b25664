// Instantiates the real row kernels with compile-time radix sequences (double).
#include "rrows.cuh"

namespace ffb {
namespace rrows {
template cudaError_t launch<double>(const TileArgs<double> &, IoKind, cudaStream_t);
template bool shape<double>(const TileArgs<double> &, IoKind, TileKernel *);
}  // namespace rrows
}  // namespace ffb
