// Instantiates the TMA column passes (tcols.cuh, wcols.cuh) in float precision.
#include "wcols_impl.cuh"

namespace ffb {

template <>
cudaError_t launch_tcols<float>(const TileArgs<float> &a, cudaStream_t s) {
  const cudaError_t e = wcols::launch_any(a, s);
  return e == cudaErrorNotSupported ? tcols::launch_any<float>(a, s) : e;
}

template <>
bool tcols_eligible<float>(int L, long long nbatch, long long G, long long ib, long long ig, long long ii, long long ob,
                          long long og, long long ok, int *threads, size_t *smem) {
  return tcols::eligible<float>(L, nbatch, G, ib, ig, ii, ob, og, ok, threads, smem);
}

template <>
bool wide_columns<float>(const TileArgs<float> &a, int *threads, size_t *smem) {
  return wcols::shape_any(a, threads, smem);
}

template <>
long long tcols_wait_failures<float>() {
#ifndef FFB_HOST_EMULATION
  int v = 0, w = 0;
  if (cudaMemcpyFromSymbol(&v, tcols::g_tcols_wait_failures, sizeof(int)) != cudaSuccess) return -1;
  if (cudaMemcpyFromSymbol(&w, wcols::g_wcols_wait_failures, sizeof(int)) != cudaSuccess) return -1;
  return (long long)v + w;
#else
  return 0;
#endif
}

}  // namespace ffb
